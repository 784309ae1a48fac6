// das_adj.cu -- the DAS adjoint (transposeDelayAndSumMex.cpp:67-97) for
// batches: lanes over instances.
//
// A pixel at travel time tau receives, from one detector, the tri taps of its
// sinogram row -- a piecewise linear function v(tau) of the row with knots at
// b, b + p1 and b + p2 of every sample b (p1, p2 = r - F and F + 1 - r in
// order: where the outermost taps enter and leave).  Per detector a CTA
// tabulates the knots of its 32 x 32 pixel block's span in shared memory,
// [knot][instance], and every (pixel, instance) interpolates between two
// neighbouring rows: acc += (1 - g) K[j] + g K[j + 1].
//
// The lanes of a pixel hold NI instances, four each, so a row read is
// NI x 4 contiguous bytes: a 128-bit load of a warp takes 4 shared wavefronts
// at NI = 32 and 6 at NI = 16 (two random rows per 8 lanes), where the table
// with one or two instances per thread (k_das_adj4: lanes over pixels, random
// 16-byte rows) paid about 10 for a quarter of the values.  (pixel, detector) pairs come as 4 bytes, knot row
// and g in fixed point, decoded once per 4 NI values.  Measured at batch 64,
// 128 x 128 px, 256 detectors: 329 us (k_das_adj4) -> 271 us (NI = 32).
//
// Bound: shared-memory wavefronts of the row reads, then the issue slots of
// the decode and of the knot table.  Every knot comes from its own window of
// samples, as in k_das_adj4: sums that run along the samples (12 operations per
// knot triple instead of 4F, 211 us) carry a NaN or a
// spike's rounding to pixels whose taps do not meet it.
//
// For calls of the operator itself.  The iterative solves keep k_das_adj4
// (apply_transpose): they amplify a last bit to 1e-3 of an image's rms at
// single pixels, so their A^T keeps one order of its sums.
#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"

namespace msot {

constexpr int A5_SIDE = 32, A5_PIX = A5_SIDE * A5_SIDE;
template <int NI> constexpr int a5_threads = NI == 32 ? 512 : 256;
// seg rows of NI + 2 words: even, for the knots' 8-byte loads, and staging
// stores along t meet each bank twice only
constexpr int A5_PAD = 2;
constexpr int A5_MIN_BATCH = 5;
constexpr int A5_RUN = 4;  // buckets that a thread tabulates from one window

struct Adj5Const {
    float inv_r, ce1;       // 1 / r, (r - F) / r
    float q1, cl;           // knot p1 = U + q1 V + cl s[b - F]
    float q2, ch;           // knot p2 = U + q2 V + ch s[b + F + 1]
    int rowbits;            // entry: g in the top 32 - rowbits bits, row below
};

static Adj5Const adj5_const(const Plan &pl) {
    const double r = pl.radius, a = r - pl.F, b = pl.F + 1 - r;
    const double p1 = std::min(a, b), p2 = std::max(a, b);
    Adj5Const c;
    c.inv_r = (float)(1.0 / r);
    c.ce1 = (float)(a / r);
    c.q1 = (float)(p1 / r);
    c.q2 = (float)(p2 / r);
    c.cl = (float)(std::max(0.0, a - p1) / r);
    c.ch = (float)(std::max(0.0, p2 - b) / r);
    c.rowbits = pl.adj5_rowbits;
    return c;
}

// span of every (32 x 32 sub-block, detector) from the 64 x 64 block table;
// sub = 4 block + 2 (z half) + (x half)
__device__ __forceinline__ int32_t a5_tau(const int32_t *btau, int sub, int D, int d, int q) {
    const int ix = (sub & 1) * 32 + q / A5_SIDE, iz = ((sub >> 1) & 1) * 32 + q % A5_SIDE;
    return btau[((size_t)(sub >> 2) * D + d) * BLK + (size_t)(ix >> 2) * BLK_THREADS +
                (ix & 3) * BLK_Z + iz];
}

__global__ void __launch_bounds__(256) k_adj5_span(const int32_t *__restrict__ btau, int D,
                                                   int fb, int2 *__restrict__ span,
                                                   int *__restrict__ most) {
    const int sub = blockIdx.y, d = blockIdx.x;
    int lo = INT32_MAX, hi = INT32_MIN;
    for (int q = threadIdx.x; q < A5_PIX; q += 256) {
        const int32_t tau = a5_tau(btau, sub, D, d, q);
        if (tau == TAU_PAD) continue;
        lo = min(lo, tau >> fb);
        hi = max(hi, tau >> fb);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    __shared__ int slo[8], shi[8];
    if ((threadIdx.x & 31) == 0) slo[threadIdx.x >> 5] = lo, shi[threadIdx.x >> 5] = hi;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) lo = min(lo, slo[k]), hi = max(hi, shi[k]);
        span[(size_t)sub * D + d] = hi >= lo ? make_int2(lo, hi) : make_int2(0, -1);
        if (hi >= lo) atomicMax(most, hi - lo + 1);
    }
}

__global__ void __launch_bounds__(256) k_adj5_entries(const int32_t *__restrict__ btau, int D,
                                                      int fb, double p1, double p2, int rowbits,
                                                      const int2 *__restrict__ span,
                                                      uint32_t *__restrict__ ent) {
    const int sub = blockIdx.y, d = blockIdx.x;
    const int lo = span[(size_t)sub * D + d].x;
    const double gs = (double)(1u << (32 - rowbits - 1)) * 2.0;
    for (int q = threadIdx.x; q < A5_PIX; q += 256) {
        const int32_t tau = a5_tau(btau, sub, D, d, q);
        uint32_t e = 0;
        if (tau != TAU_PAD) {
            const double f = (double)(tau & ((1 << fb) - 1)) / (double)(1 << fb);
            const int c = (f >= p1) + (f >= p2);
            const double a = c == 0 ? 0.0 : c == 1 ? p1 : p2, b = c == 0 ? p1 : c == 1 ? p2 : 1.0;
            const double g = (f - a) / (b - a) * gs;  // b > a: f lies in [a, b)
            const uint32_t gq = (uint32_t)fmin(rint(g), gs - 1.0);
            e = gq << rowbits | (uint32_t)((((tau >> fb) - lo) * 3) + c);
        }
        ent[((size_t)sub * D + d) * A5_PIX + q] = e;
    }
}

// Grid (sub-block, instance tile, detector group); instances w0 + 0 .. NI - 1,
// those past W read as zero and are not stored.
template <int NI, int F>
__global__ void __launch_bounds__(a5_threads<NI>, NI == 32 ? 1 : 2) k_das_adj5(
    const uint32_t *__restrict__ ent, const int2 *__restrict__ bspan,
    const float *__restrict__ s, float *__restrict__ part, int nx, int nz, int nbx, int D,
    int T, int W, Adj5Const cst, int seg_rows, int knot_rows, int det_per_group,
    size_t part_stride) {
    constexpr int A5_THREADS = a5_threads<NI>;
    constexpr int LPG = NI / 4;                  // lanes per pixel
    constexpr int NG = A5_THREADS / LPG;         // pixels in flight
    constexpr int PPG = A5_PIX / NG;             // pixels per lane group
    constexpr int RS = NI + A5_PAD;              // words per seg row
    constexpr int NP = NI / 2, NRUN = A5_THREADS / NP;  // runs of the knot table
    extern __shared__ __align__(16) float a5_smem[];
    float *K = a5_smem;                          // [knot_rows][NI]
    float *seg0 = K + (size_t)knot_rows * NI;    // [2][seg_rows][RS]
    const int sub = blockIdx.x, w0 = blockIdx.y * NI, grp = blockIdx.z;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int d_begin = grp * det_per_group, d_end = min(D, d_begin + det_per_group);
    const uint32_t rowmask = (1u << cst.rowbits) - 1u, gmask = (0xffffffffu << cst.rowbits) >> 9;
    float2 acc[PPG][2];
#pragma unroll
    for (int i = 0; i < PPG; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);

    // seg row k = sample span.x - F + k; zero outside [0, T) and past W
    auto stage = [&](int d, int buf) {
        const int2 sp = __ldg(bspan + (size_t)sub * D + d);
        const int n = sp.y - sp.x + 1 + 2 * F + 3;
        if (sp.y < sp.x) return;
        float *seg = seg0 + (size_t)buf * seg_rows * RS;
        const bool inside = sp.x - F >= 0 && sp.x - F + n <= T && w0 + NI <= W;
        for (int w = warp; w < NI; w += A5_THREADS / 32) {
            const float *src = s + ((size_t)min(w0 + w, W - 1) * D + d) * T;
            if (inside) {
                uint32_t dst = smem_u32(seg + lane * RS + w);
                src += sp.x - F + lane;
                for (int k = lane; k < n; k += 32, src += 32, dst += 32 * RS * 4)
                    cp_async4(dst, src);
                continue;
            }
            const bool in = w0 + w < W;
            for (int k = lane; k < n; k += 32) {
                const int tt = sp.x - F + k;
                const bool ok = in && tt >= 0 && tt < T;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                                 smem_u32(seg + k * RS + w)),
                             "l"(src + (ok ? tt : 0)), "r"(ok ? 4 : 0)
                             : "memory");
            }
        }
    };
    if (d_begin < d_end) stage(d_begin, 0);
    const int run = t / NP, inst = t % NP * 2;
    const int grp_px = t / LPG, l4 = (t % LPG) * 4;
    for (int d = d_begin; d < d_end; ++d) {
        const int buf = (d - d_begin) & 1;
        const int2 sp = __ldg(bspan + (size_t)sub * D + d);
        const int nb = sp.y - sp.x + 1;  // uniform across the CTA
        cp_async_wait_all();
        __syncthreads();  // seg[buf] is complete; the last gather is done with K
        if (d + 1 < d_end) stage(d + 1, buf ^ 1);
        if (nb <= 0) continue;
        {
            // knots of buckets 0 .. nb (the last one's first row closes the
            // table), two instances side by side in packed arithmetic
            constexpr int NWIN = 2 * F + 1 + A5_RUN;
            auto two = [](float v) { return make_float2(v, v); };
            for (int b0 = run * A5_RUN; b0 <= nb; b0 += NRUN * A5_RUN) {
                const float *g = seg0 + (size_t)buf * seg_rows * RS + inst + (size_t)b0 * RS;
                float2 win[NWIN];  // win[F + j]: sample b0 + j
#pragma unroll
                for (int j = 0; j < NWIN; ++j)
                    win[j] = *reinterpret_cast<const float2 *>(g + j * RS);
                float *row = K + (size_t)3 * b0 * NI + inst;
#pragma unroll
                for (int r = 0; r < A5_RUN; ++r, row += 3 * NI) {
                    if (b0 + r > nb) break;
                    float2 U = two(0.f), V0 = U, V1 = U;
#pragma unroll
                    for (int k = F - 1; k >= 0; --k) {
                        const float2 v = win[r + F - k];
                        U = ffma2(two(1.f - (float)k * cst.inv_r), v, U);
                        V0 = fadd2(V0, v);
                    }
#pragma unroll
                    for (int k = F; k >= 1; --k) {
                        const float2 v = win[r + F + k];
                        U = ffma2(two(1.f - (float)k * cst.inv_r), v, U);
                        V1 = fadd2(V1, v);
                    }
                    const float2 V = ffma2(V0, two(-1.f), V1), sl = win[r],
                                 sh = win[r + 2 * F + 1];
                    float2 *o = reinterpret_cast<float2 *>(row);
                    o[0] = ffma2(two(cst.ce1), sl, U);
                    o[NP] = ffma2(two(cst.q1), V, ffma2(two(cst.cl), sl, U));
                    o[2 * NP] = ffma2(two(cst.q2), V, ffma2(two(cst.ch), sh, U));
                }
            }
        }
        __syncthreads();
        const uint32_t *e = ent + ((size_t)sub * D + d) * A5_PIX + grp_px;
        constexpr int CH = PPG < 8 ? PPG : 8;
#pragma unroll
        for (int i0 = 0; i0 < PPG; i0 += CH) {
            uint32_t q[CH];
#pragma unroll
            for (int i = 0; i < CH; ++i) q[i] = __ldg(e + (i0 + i) * NG);
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                // 1 + g in the mantissa
                const float m = __uint_as_float(((q[i] >> 9) & gmask) | 0x3f800000u);
                const float g = m - 1.f, h = 2.f - m;
                const float4 *row =
                    reinterpret_cast<const float4 *>(K + (q[i] & rowmask) * NI + l4);
                const float4 a = row[0], b = row[LPG];
                const float2 g2 = make_float2(g, g), h2 = make_float2(h, h);
                acc[i0 + i][0] = ffma2(h2, make_float2(a.x, a.y), acc[i0 + i][0]);
                acc[i0 + i][1] = ffma2(h2, make_float2(a.z, a.w), acc[i0 + i][1]);
                acc[i0 + i][0] = ffma2(g2, make_float2(b.x, b.y), acc[i0 + i][0]);
                acc[i0 + i][1] = ffma2(g2, make_float2(b.z, b.w), acc[i0 + i][1]);
            }
        }
    }
    const size_t P = (size_t)nx * nz;
    float *dst = part + (size_t)grp * part_stride;
    const int blk = sub >> 2;
    const int x0 = (blk % nbx) * BLK_X + (sub & 1) * 32;
    const int z0 = (blk / nbx) * BLK_Z + ((sub >> 1) & 1) * 32;
#pragma unroll
    for (int i = 0; i < PPG; ++i) {
        const int q = i * NG + grp_px;
        const int ix = x0 + q / A5_SIDE, iz = z0 + q % A5_SIDE;
        if (ix >= nx || iz >= nz) continue;
        float *o = dst + (size_t)(w0 + l4) * P + (size_t)ix * nz + iz;
        const float v[4] = {acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (w0 + l4 + j < W) o[(size_t)j * P] = v[j];
    }
}

static size_t adj5_smem(const Plan &pl, int ni) {
    return ((size_t)(3 * pl.adj5_span_max + 4) * ni +
            (size_t)2 * (pl.adj5_span_max + 2 * pl.F + 2 + A5_RUN) * (ni + A5_PAD)) *
           sizeof(float);
}

// instances per tile: the widest that W fills to more than half and whose
// tables leave two CTAs per SM (one of twice the threads at 32); 0: none does
static int adj5_ni(const Plan &pl, int W) {
    int ni = W > 16 && (W + 31) / 32 * 32 - W < 16 ? 32 : W > 8 ? 16 : 8;
    while (ni >= 8 && adj5_smem(pl, ni) > (ni == 32 ? 222 : 110) * 1024) ni /= 2;
    return ni >= 8 ? ni : 0;
}

int adj5_build(Plan &p, size_t &bytes) {
    const int subs = 4 * p.n_blk;
    // k_das_adj4 serves such plans: smaller batches never take the kernel
    if (p.max_batch < A5_MIN_BATCH || subs > 65535) return MSOT_OK;
    MSOT_MALLOC_TRY(cudaMalloc(&p.adj5_span, sizeof(int2) * (size_t)subs * p.D));
    bytes += sizeof(int2) * (size_t)subs * p.D;
    int *most = nullptr;
    MSOT_MALLOC_TRY(cudaMalloc(&most, sizeof(int)));
    cudaMemset(most, 0, sizeof(int));
    const dim3 grid(p.D, subs);
    KLAUNCH(k_adj5_span<<<grid, 256>>>(p.blk_tau, p.D, p.frac_bits, p.adj5_span, most));
    int span = 0;
    const cudaError_t e = cudaMemcpy(&span, most, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(most);
    MSOT_CUDA_TRY(e);
    int bits = 1;
    while ((1 << bits) < 3 * span + 1) ++bits;
    // rows beyond 11 bits would leave g less than the travel times' resolution
    if (bits > 11) return MSOT_OK;
    p.adj5_rowbits = bits;
    p.adj5_span_max = span;
    if (!adj5_ni(p, A5_MIN_BATCH)) return MSOT_OK;  // no tile's tables fit shared memory
    const size_t n = (size_t)subs * p.D * A5_PIX;
    MSOT_MALLOC_TRY(cudaMalloc(&p.adj5_ent, sizeof(uint32_t) * n));
    bytes += sizeof(uint32_t) * n;
    const double a = p.radius - p.F, b = p.F + 1 - p.radius;
    KLAUNCH(k_adj5_entries<<<grid, 256>>>(p.blk_tau, p.D, p.frac_bits, std::min(a, b),
                                          std::max(a, b), bits, p.adj5_span, p.adj5_ent));
    MSOT_LAUNCH_CHECK();
    return MSOT_OK;
}

template <int NI, int F>
static int adj5_launch(const Plan &pl, const float *raw, float *part, int W, int groups, int dpg,
                       size_t stride, cudaStream_t st) {
    const size_t smem = adj5_smem(pl, NI);
    int rc = set_smem(k_das_adj5<NI, F>, smem);
    if (rc) return rc;
    const dim3 grid(4 * pl.n_blk, div_up(W, NI), groups);
    KLAUNCH(k_das_adj5<NI, F><<<grid, a5_threads<NI>, smem, st>>>(
        pl.adj5_ent, pl.adj5_span, raw, part, pl.nx, pl.nz, pl.n_blk_x, pl.D, pl.T, W,
        adj5_const(pl), pl.adj5_span_max + 2 * pl.F + 2 + A5_RUN, 3 * pl.adj5_span_max + 4, dpg, stride));
    MSOT_LAUNCH_CHECK();
    return MSOT_OK;
}

template <int NI>
static int adj5_f(const Plan &pl, const float *raw, float *part, int W, int groups, int dpg,
                  size_t stride, cudaStream_t st) {
    switch (pl.F) {
        case 0: return adj5_launch<NI, 0>(pl, raw, part, W, groups, dpg, stride, st);
        case 1: return adj5_launch<NI, 1>(pl, raw, part, W, groups, dpg, stride, st);
        case 2: return adj5_launch<NI, 2>(pl, raw, part, W, groups, dpg, stride, st);
        case 3: return adj5_launch<NI, 3>(pl, raw, part, W, groups, dpg, stride, st);
        case 4: return adj5_launch<NI, 4>(pl, raw, part, W, groups, dpg, stride, st);
        case 5: return adj5_launch<NI, 5>(pl, raw, part, W, groups, dpg, stride, st);
        case 6: return adj5_launch<NI, 6>(pl, raw, part, W, groups, dpg, stride, st);
        case 7: return adj5_launch<NI, 7>(pl, raw, part, W, groups, dpg, stride, st);
        default: return adj5_launch<NI, 8>(pl, raw, part, W, groups, dpg, stride, st);
    }
}

// whether k_das_adj5 beats k_das_adj4 for W instances: odd batches (one instance
// per CTA there) from 5 up, others where three quarters of the instance tiles
// are filled.  k_das_adj4 / k_das_adj5 in us for 6, 8, 12, 18, 24, 64 images of
// 128 x 128 px: 49 / 55, 50 / 54, 84 / 80, 100 / 128, 148 / 133, 329 / 271; 200 x 200 px,
// 6, 8, 10, 16, 28: 123 / 128, 166 / 126, 214 / 206, 276 / 207, 403 / 366; 400 x 400 px,
// 512 detectors, 5, 6, 8, 13: 1083 / 665, 523 / 668, 721 / 660, 2277 / 950
bool adj5_usable(const Plan &pl, int W) {
    const int ni = pl.adj5_ent && W >= A5_MIN_BATCH ? adj5_ni(pl, W) : 0;
    return ni && (W % 2 || (W >= 8 && 4 * W >= 3 * ni * div_up(W, ni)));
}

int launch_das_adjoint5(const Plan &pl, const float *raw, float *x, int W, float scale,
                        cudaStream_t st) {
    const int ni = adj5_ni(pl, W);
    // detector groups: the fewest that come close to filling whole waves of two
    // CTAs per SM, one at NI = 32 (each group writes a partial image)
    const int base = 4 * pl.n_blk * div_up(W, ni), slots = (ni == 32 ? 1 : 2) * sm_count();
    const int most = std::max(1, std::min({pl.adj_groups_max * pl.max_batch / W, pl.D, 32}));
    int groups = 1;
    double best = 0.0;
    for (int g = 1; g <= most; ++g) {
        const int dpg = div_up(pl.D, g), n = base * div_up(pl.D, dpg);
        const double eff = (double)base * pl.D / ((double)div_up(n, slots) * slots * dpg);
        if (eff > best * 1.05) best = eff, groups = g;
    }
    const int dpg = div_up(pl.D, groups);
    groups = div_up(pl.D, dpg);
    const size_t stride = (size_t)W * pl.P;
    const int rc = ni == 32   ? adj5_f<32>(pl, raw, pl.scr_part, W, groups, dpg, stride, st)
                   : ni == 16 ? adj5_f<16>(pl, raw, pl.scr_part, W, groups, dpg, stride, st)
                            : adj5_f<8>(pl, raw, pl.scr_part, W, groups, dpg, stride, st);
    if (rc) return rc;
    return sum_parts(pl.scr_part, x, stride, groups, scale, st);
}

}  // namespace msot

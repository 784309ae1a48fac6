// das_fwd_lanes.cu -- the DAS forward (forwardDelayAndSumMex.cpp:72-103) for
// batches: lanes over instances.
//
// The same bucket moments and filter as k_das_fwd3 (das_fwd.cuh), but a bucket
// belongs to a group of NI / 4 lanes that hold four instances each, so one
// pixel's NI values are one 128-byte (NI = 32) or 64-byte load.  The SM's L1
// serves one line per cycle: k_das_fwd3's lanes read 32 bytes of 32 different
// lines (58 M wavefronts per launch at batch 64, the pipe 77 % busy), here a
// line carries NI x 4 bytes of it.  A CTA takes the same 64 buckets of DG
// neighbouring detectors at once, whose arcs cross the same pixels, so that
// L1 halves (DG = 2) or quarters the L2 traffic.  The entries come eight per
// load and group (CSR order) and are handed round by shuffles.
// Measured at batch 64, 128 x 128 px, 256 detectors: 245 us (k_das_fwd3, 8
// instances per CTA) -> 184 us; at 200 x 200 px,
// batch 28, 350 -> 180 us.
#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"

namespace msot {

constexpr int F6_THREADS = 256, F6_NB = 64;  // buckets per detector and CTA
template <int NI> constexpr int f6_dg = 64 / NI;                    // detectors per CTA
template <int NI> constexpr int f6_row = f6_dg<NI> * F6_NB + 32 / NI;  // conflict-free stores

template <int NI, int F>
__global__ void __launch_bounds__(F6_THREADS, F <= 2 ? 2 : 3) k_das_fwd6(
    const int32_t *__restrict__ off, const int2 *__restrict__ ent,
    const float *__restrict__ xpm, float *__restrict__ raw, int P, int D, int T, int W, int fb,
    float inv_r, float ce1, float ce2, float scale, const int2 *__restrict__ skip) {
    constexpr int LPG = NI / 4, NG = F6_THREADS / LPG, DG = f6_dg<NI>, ROW = f6_row<NI>;
    constexpr int PER = NG / DG;  // buckets of a detector in flight: 16
    // Pixels in flight per lane group.  Coarse radii (F <= 2, long lists) take
    // eight at two CTAs per SM, which leaves more of L1 to the pixels: 13 images
    // of 400 x 400 px, 512 detectors 962 -> 601 us; lists of a dozen entries
    // lose to the padding (64 images of 128 x 128 px 208 -> 233 us with eight).
    constexpr int TB = F6_NB - 2 * F - 2, CH = 8, BT = F <= 2 ? 8 : 4;
    extern __shared__ float mom[];  // [4][NI][ROW], bucket fastest
    const int d0 = blockIdx.y * DG, w0 = blockIdx.z * NI;
    const int t0 = blockIdx.x * TB, b_lo = t0 - F - 1;
    const int lane = threadIdx.x & 31, l = threadIdx.x % LPG;
    const int bi = threadIdx.x % F6_NB, di = threadIdx.x / F6_NB;
    {
        const int d = d0 + di % DG;
        const int32_t *o = off + (size_t)min(d, D - 1) * (T + 1);
        const int bl = max(b_lo, 0), bh = min(b_lo + F6_NB, T);
        const bool some = d < D && bl < bh && __ldg(o + bl) != __ldg(o + bh);
        if (!__syncthreads_or(some)) {
            // no pixel of these detectors falls in the CTA's buckets
            if (d >= D) return;
            if (skip) {  // wholly outside the support: nobody reads it
                const int2 sup = __ldg(skip + d);
                if (t0 >= sup.y || t0 + TB <= sup.x) return;
            }
            const int t = t0 + bi;
            if (bi < TB && t < T)
                for (int i = di / DG; i < NI && w0 + i < W; i += F6_THREADS / F6_NB / DG)
                    raw[((size_t)(w0 + i) * D + d) * T + t] = 0.f;
            return;
        }
    }
    {
        const int grp = threadIdx.x / LPG, dd = grp / PER, d = min(d0 + dd, D - 1);
        const bool have = d0 + dd < D;
        const int32_t *o = off + (size_t)d * (T + 1);
        const int2 *e = ent + (size_t)d * P;
        const float4 *x = reinterpret_cast<const float4 *>(xpm) + (size_t)blockIdx.z * P * LPG + l;
        const int mask = (1 << fb) - 1;
        const float step = __int_as_float((127 - fb) << 23);  // 2^-fb
#pragma unroll 1
        for (int r = 0; r < F6_NB; r += PER) {
            const int bk = r + grp % PER, b = b_lo + bk;
            int j0 = 0, n = 0;
            if (have && b >= 0 && b < T) {
                j0 = __ldg(o + b);
                n = __ldg(o + b + 1) - j0;
            }
            const int most = __reduce_max_sync(0xffffffffu, n);
            float2 m0[2], m1[2], m2[2], m3[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) m0[k] = m1[k] = m2[k] = m3[k] = make_float2(0.f, 0.f);
            // lane l holds the entries l, l + LPG, .. of the current chunk
            int2 q[CH / LPG];
            auto fetch = [&](int c) {
#pragma unroll
                for (int k = 0; k < CH / LPG; ++k) {
                    // the address stays inside the table where the list has ended
                    const int j = c + k * LPG + l;
                    q[k] = __ldg(e + min(j0 + min(j, max(n - 1, 0)), P - 1));
                    if (j >= n) q[k] = make_int2(0, -1);
                }
            };
            fetch(0);
            for (int c = 0; c < most; c += CH) {
                int pix[CH / LPG];
                float fr[CH / LPG];
#pragma unroll
                for (int k = 0; k < CH / LPG; ++k) {
                    pix[k] = q[k].y;
                    fr[k] = (float)(q[k].x & mask) * step;
                }
                if (c + CH < most) fetch(c + CH);
#pragma unroll
                for (int h = 0; h < CH; h += BT) {
                    if (c + h >= most) break;  // uniform in the warp
                    float4 v[BT];
                    float f[BT];
#pragma unroll
                    for (int k = 0; k < BT; ++k) {
                        const int p =
                            __shfl_sync(0xffffffffu, pix[(h + k) / LPG], (h + k) % LPG, LPG);
                        f[k] = __shfl_sync(0xffffffffu, fr[(h + k) / LPG], (h + k) % LPG, LPG);
                        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (p >= 0) v[k] = __ldg(x + (size_t)max(p, 0) * LPG);
                    }
#pragma unroll
                    for (int k = 0; k < BT; ++k) {
                        const float e1 = fmaxf(0.f, fmaf(-f[k], inv_r, ce1));
                        const float e2 = fmaxf(0.f, fmaf(f[k], inv_r, -ce2));
                        const float2 a = make_float2(v[k].x, v[k].y),
                                     bb = make_float2(v[k].z, v[k].w);
                        const float2 ff = make_float2(f[k], f[k]), ea = make_float2(e1, e1),
                                     eb = make_float2(e2, e2);
                        m0[0] = fadd2(m0[0], a);
                        m0[1] = fadd2(m0[1], bb);
                        m1[0] = ffma2(ff, a, m1[0]);
                        m1[1] = ffma2(ff, bb, m1[1]);
                        m2[0] = ffma2(ea, a, m2[0]);
                        m2[1] = ffma2(ea, bb, m2[1]);
                        m3[0] = ffma2(eb, a, m3[0]);
                        m3[1] = ffma2(eb, bb, m3[1]);
                    }
                }
            }
            float *m = mom + (size_t)(4 * l) * ROW + dd * F6_NB + bk;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                m[(0 * NI + 2 * k) * ROW] = m0[k].x;
                m[(0 * NI + 2 * k + 1) * ROW] = m0[k].y;
                m[(1 * NI + 2 * k) * ROW] = m1[k].x;
                m[(1 * NI + 2 * k + 1) * ROW] = m1[k].y;
                m[(2 * NI + 2 * k) * ROW] = m2[k].x;
                m[(2 * NI + 2 * k + 1) * ROW] = m2[k].y;
                m[(3 * NI + 2 * k) * ROW] = m3[k].x;
                m[(3 * NI + 2 * k + 1) * ROW] = m3[k].y;
            }
        }
    }
    __syncthreads();
    // the filter over the moments, the chain of k_das_fwd3
    const int d = d0 + di % DG, t = t0 + bi;
    if (bi >= TB || t >= T || d >= D) return;
    const int base = (di % DG) * F6_NB + bi + F + 1;  // bucket t
#pragma unroll 4
    for (int i = di / DG; i < NI; i += F6_THREADS / F6_NB / DG) {
        if (w0 + i >= W) break;
        const float *M0 = mom + (size_t)(0 * NI + i) * ROW + base;
        const float *M1 = mom + (size_t)(1 * NI + i) * ROW + base;
        float acc = mom[(size_t)(2 * NI + i) * ROW + base + F] +
                    mom[(size_t)(3 * NI + i) * ROW + base - F - 1];
#pragma unroll
        for (int k = -(F - 1); k <= F; ++k) {
            acc = fmaf(1.f - (float)(k < 0 ? -k : k) * inv_r, M0[-k], acc);
            acc = fmaf(k <= 0 ? -inv_r : inv_r, M1[-k], acc);
        }
        raw[((size_t)(w0 + i) * D + d) * T + t] = acc * scale;
    }
}

template <int NI, int F>
static int fwd6_launch(const Plan &pl, const float *xpm, float *raw, int W, float scale,
                       const int2 *skip, cudaStream_t st) {
    constexpr int TB = F6_NB - 2 * F - 2;
    constexpr size_t smem = (size_t)4 * NI * f6_row<NI> * sizeof(float);
    int rc = set_smem(k_das_fwd6<NI, F>, smem);
    if (rc) return rc;
    const dim3 grid(div_up(pl.T, TB), div_up(pl.D, f6_dg<NI>), div_up(W, NI));
    KLAUNCH(k_das_fwd6<NI, F><<<grid, F6_THREADS, smem, st>>>(
        pl.fwd_off, pl.fwd_ent, xpm, raw, pl.P, pl.D, pl.T, W, pl.frac_bits, pl.inv_r, pl.ce1,
        pl.ce2, scale, skip));
    MSOT_LAUNCH_CHECK();
    return MSOT_OK;
}

template <int NI>
static int fwd6_f(const Plan &pl, const float *xpm, float *raw, int W, float scale,
                  const int2 *skip, cudaStream_t st) {
    switch (pl.F) {
        case 0: return fwd6_launch<NI, 0>(pl, xpm, raw, W, scale, skip, st);
        case 1: return fwd6_launch<NI, 1>(pl, xpm, raw, W, scale, skip, st);
        case 2: return fwd6_launch<NI, 2>(pl, xpm, raw, W, scale, skip, st);
        case 3: return fwd6_launch<NI, 3>(pl, xpm, raw, W, scale, skip, st);
        case 4: return fwd6_launch<NI, 4>(pl, xpm, raw, W, scale, skip, st);
        case 5: return fwd6_launch<NI, 5>(pl, xpm, raw, W, scale, skip, st);
        case 6: return fwd6_launch<NI, 6>(pl, xpm, raw, W, scale, skip, st);
        case 7: return fwd6_launch<NI, 7>(pl, xpm, raw, W, scale, skip, st);
        default: return fwd6_launch<NI, 8>(pl, xpm, raw, W, scale, skip, st);
    }
}

int launch_das_forward_lanes(const Plan &pl, const float *xpm, float *raw, int W, int wt,
                             float scale, const int2 *skip, cudaStream_t st) {
    return wt == 32 ? fwd6_f<32>(pl, xpm, raw, W, scale, skip, st)
                    : fwd6_f<16>(pl, xpm, raw, W, scale, skip, st);
}

}  // namespace msot

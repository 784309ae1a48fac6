// analytic.cu -- the reference's analytic reconstructors on the GPU.
//
//   msot_dmas_cf            <- reconstruction_backprojection/dmas_cf.m:19-107
//   msot_backproject_waveeq <- reconstruction_backprojection/backproject_waveeq.m:1-50
//
// Both index the sinogram at the nearest sample of the pixel-to-detector
// travel time, round((|x_p - x_d| / c - t_1) fs + 1) (dmas_cf.m:69-74,
// backproject_waveeq.m:36-41).  That index is the FP64 reference's: near a rounding
// tie it is computed in FP64 with every operation rounded separately (no
// contraction into FMA), elsewhere an FP32 estimate settles it; an index
// outside the sinogram, where MATLAB raises an error, is reported as
// MSOT_ERANGE.  Sums over detectors and samples are pairs of floats
// (twofloat.cuh, about 48 bits), in FP64 where they leave FP32's range; the
// results' errors against 64 bits are those of FP64 sums to every digit
// measured (filtered 3.3e-6, waveeq 1.0e-5, the four of dmas_cf 0.6 to 2.3e-6
// at 78, 128 and 200 px): the FP32 inputs and outputs make them.

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "twofloat.cuh"

namespace msot {

// idx[d][p] = 0-based nearest sample index of pixel p for detector d.  The FP64
// expression (square root, division) decides only where it can: an FP32
// estimate (coordinates xf, zf, det rounded to FP32) whose error is below
// `tol` settles every value that is further
// than that from a rounding tie (all but about one pair in 50 at 40 MHz),
// the others take the FP64 path.  4.2 M pairs: 219 -> 40 us.
__global__ void k_nearest_index(const double *__restrict__ cosa, const double *__restrict__ sina,
                                const double *__restrict__ xv, const double *__restrict__ zv,
                                const float *__restrict__ xf, const float *__restrict__ zf,
                                const float2 *__restrict__ det, float per_m, float off, int nx, int nz, int D, double R, double c, double fs,
                                double acq1, int T, float tol, int32_t *__restrict__ idx,
                                int *err) {
    const int P = nx * nz;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int d = blockIdx.y;
    if (p >= P) return;
    const int ix = p / nz, iz = p - ix * nz;
    const float2 xz = make_float2(__ldg(xf + ix), __ldg(zf + iz)), cr = __ldg(det + d);
    const float fx = xz.x - cr.x, fz = xz.y - cr.y;
    const float est = fmaf(sqrtf(fmaf(fx, fx, fz * fz)), per_m, off);
    const float half = est + 0.5f, lo = floorf(half);
    long i;
    if (half - lo > tol && half - lo < 1.f - tol && est > 1.f && est < 8388608.f) {
        i = (long)lo - 1;
    } else {
        const double dx = __dadd_rn(xv[ix], -__dmul_rn(cosa[d], R));
        const double dz = __dadd_rn(zv[iz], -__dmul_rn(sina[d], R));
        const double dist = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dz, dz)));
        const double v =
            __dadd_rn(__dmul_rn(__dadd_rn(__ddiv_rn(dist, c), -acq1), fs), 1.0);
        i = (long)round(v) - 1;
    }
    if (i < 0 || i >= T) {
        atomicOr(err, 1);
        i = i < 0 ? 0 : T - 1;
    }
    idx[(size_t)d * P + p] = (int32_t)i;
}

__global__ void k_max_abs(const float *__restrict__ x, size_t n, unsigned int *out) {
    float m = 0.f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        m = fmaxf(m, fabsf(x[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));  // m >= 0: order preserved
}

// Pixel tiles of the two gathers below: a CTA's 256 pixels (32 along z x 8
// along x) read a few hundred neighbouring samples of one detector row, which
// L1 then serves; AN_FR frames per thread share each index load.
constexpr int AN_TZ = 32, AN_TX = 8, AN_THREADS = AN_TZ * AN_TX, AN_FR = 4;

// dmas_cf.m:63-105: per pixel and frame the four detector sums, each as a
// pair of floats (twofloat.cuh) over samples scaled by a power of two (exact);
// the square roots get one Newton correction as their tail.  64 frames of
// 128 x 128 px, 256 detectors: 7.37 ms with FP64 sums and roots (bound by the
// FP64 pipe) -> 0.48 ms (the gathers).
__global__ void __launch_bounds__(AN_THREADS, 3) k_dmas_cf(
    const float *__restrict__ sig, const int32_t *__restrict__ idx,
    const unsigned int *__restrict__ maxbits, int nx, int nz, int W, int D, int T,
    float *__restrict__ o_dmascf, float *__restrict__ o_dmas, float *__restrict__ o_cf,
    float *__restrict__ o_das) {
    const int iz = blockIdx.x * AN_TZ + threadIdx.x % AN_TZ;
    const int ix = blockIdx.y * AN_TX + threadIdx.x / AN_TZ;
    if (ix >= nx || iz >= nz) return;
    const size_t P = (size_t)nx * nz, p = (size_t)ix * nz + iz;
    const int w0 = blockIdx.z * AN_FR;
    const float mx = __uint_as_float(*maxbits);
    // the power of two that brings the maximum to about 1
    const float sc = ldexpf(1.f, -max(-120, min(120, (int)(*maxbits >> 23) - 127)));
    const float *s[AN_FR];
#pragma unroll
    for (int f = 0; f < AN_FR; ++f) s[f] = sig + (size_t)min(w0 + f, W - 1) * D * T;
    Sum2 sos[AN_FR / 2], sqs[AN_FR / 2], num[AN_FR / 2], den[AN_FR / 2];
#pragma unroll
    for (int f = 0; f < AN_FR / 2; ++f) {
        sos[f].zero();
        sqs[f].zero();
        num[f].zero();
        den[f].zero();
    }
    const float2 sc2 = make_float2(sc, sc), m1 = make_float2(-1.f, -1.f);
#pragma unroll 2
    for (int d = 0; d < D; ++d) {
        const size_t at = (size_t)d * T + __ldg(idx + (size_t)d * P + p);
#pragma unroll
        for (int f = 0; f < AN_FR / 2; ++f) {
            const float2 v =
                __fmul2_rn(make_float2(__ldg(s[2 * f] + at), __ldg(s[2 * f + 1] + at)), sc2);
            const float2 a = make_float2(fabsf(v.x), fabsf(v.y));
            // sign(v) sqrt(a) = q + y (a - q^2) / 2 to second order, y = 1 / sqrt(a)
            const float2 y = make_float2(rsqrtf(fmaxf(a.x, 1e-37f)), rsqrtf(fmaxf(a.y, 1e-37f)));
            const float2 q = __fmul2_rn(v, y);
            const float2 r = ffma2(__fmul2_rn(q, m1), q, a);
            const float2 hy = __fmul2_rn(y, make_float2(0.5f, 0.5f));
            const float2 t = __fmul2_rn(
                r, make_float2(copysignf(hy.x, v.x), copysignf(hy.y, v.y)));
            const float2 vv = __fmul2_rn(v, v);
            sos[f].add(a);
            sqs[f].add(q, t);
            num[f].add(v);
            den[f].add(vv, ffma2(v, v, __fmul2_rn(vv, m1)));
        }
    }
    // the reference divides the sinogram by its maximum: g undoes the power of two
    const double g = 1.0 / ((double)mx * (double)sc);
    const double gr = sqrt(g);
#pragma unroll
    for (int f = 0; f < AN_FR; ++f) {
        if (w0 + f >= W) break;
        const double ss = g * (f & 1 ? sos[f / 2].y() : sos[f / 2].x());
        const double sq = gr * (f & 1 ? sqs[f / 2].y() : sqs[f / 2].x());
        const double nu = g * (f & 1 ? num[f / 2].y() : num[f / 2].x());
        const double de = g * g * (f & 1 ? den[f / 2].y() : den[f / 2].x());
        const double dmas = 0.5 * (sq * sq - ss);
        const double cf = nu * nu / (1e-6 + (double)D * de);
        const size_t o = (size_t)(w0 + f) * P + p;
        o_dmascf[o] = (float)(dmas * cf);
        o_dmas[o] = (float)dmas;
        o_cf[o] = (float)cf;
        o_das[o] = (float)nu;
    }
}

// backproject_waveeq.m:23-24: cumtrapz(t, sig / c) ./ t per column.  With
// uniform times the trapezoids' running sum is 2 C_t - s_0 - s_t, C the
// running sum of the samples, and the factors 0.5 dt / c / t_k come from a
// table (hi, lo).  One warp per column staged in shared memory: lane l sums
// its ceil(T / 32) consecutive samples as a pair of floats, a warp scan gives
// each lane its start, a second walk writes the results, which leave
// coalesced.  Columns too long for shared memory are walked in `out`.  16384
// columns of 2030: 2.05 ms (one thread per column, FP64) -> 0.12 ms.
constexpr int CT_WARPS = 4;
__global__ void __launch_bounds__(32 * CT_WARPS) k_cumtrapz(const float *__restrict__ sig,
                                                            float *out, int cols,
                                                            int T, int ldo, int staged,
                                                            const float2 *__restrict__ fac) {
    extern __shared__ float ct_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col = blockIdx.x * CT_WARPS + warp;
    if (col >= cols) return;  // whole warp; no CTA-wide barriers below
    const int per = ((T + 31) / 32) | 1;  // odd: lanes' walks hit distinct banks
    const float *s = sig + (size_t)col * T;
    float *o = out + (size_t)col * ldo;
    float *buf = staged ? ct_smem + (size_t)warp * (32 * per) : o;
    for (int t = lane; t < T; t += 32) buf[t] = __ldg(s + t);
    __syncwarp();
    const float first = buf[0];
    __syncwarp();
    const int a = min(lane * per, T), b = min(a + per, T);
    Sum1 own;
    float big = 0.f;
    for (int t = a; t < b; ++t) {
        own.add(buf[t]);
        big = fmaxf(big, fabsf(buf[t]));
    }
    if (__any_sync(0xffffffffu, !(big * T < 1e38f))) {
        // twice the sum may leave FP32's range: the trapezoids in FP64
        double acc = 0.0;
        float prev = a > 0 && a < T ? buf[a - 1] : first;
        const float before = prev;
        for (int t = a; t < b; prev = buf[t++])
            if (t) acc += 0.5 * ((double)buf[t] + (double)prev);
        double run = acc;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, run, k);
            if (lane >= k) run += u;
        }
        run = __shfl_up_sync(0xffffffffu, run, 1);
        acc = lane ? run : 0.0;
        prev = before;
        __syncwarp();  // every lane has read its neighbour's last sample
        for (int t = a; t < b; ++t) {
            const float v = buf[t];
            if (t) acc += 0.5 * ((double)v + (double)prev);
            prev = v;
            const float2 f = __ldg(fac + t);
            buf[t] = t ? (float)(2.0 * acc * ((double)f.x + (double)f.y)) : 0.f;
        }
        __syncwarp();
        if (staged)
            for (int t = lane; t < T; t += 32) o[t] = buf[t];
        return;
    }
    // exclusive scan of the lanes' sums (FP64: five steps per column)
    double run = own.value();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += u;
    }
    run = __shfl_up_sync(0xffffffffu, run, 1);
    if (lane == 0) run = 0.0;
    Sum1 acc;
    acc.s = (float)run;
    acc.c = (float)(run - (double)acc.s);
    for (int t = a; t < b; ++t) {
        const float v = buf[t];
        acc.add(v);
        Sum1 z;  // 2 C_t - s_0 - s_t
        z.s = 2.f * acc.s;
        z.c = 2.f * acc.c;
        z.add(-v);
        z.add(-first);
        const float2 f = __ldg(fac + t);
        const float h = z.s * f.x;
        buf[t] = t ? h + (fmaf(z.s, f.x, -h) + fmaf(z.s, f.y, z.c * f.x)) : 0.f;
    }
    __syncwarp();
    if (staged)
        for (int t = lane; t < T; t += 32) o[t] = buf[t];
}

// backproject_waveeq.m:27: convn(sig, psf, 'same') / sum(psf) over (T, D) of
// each wavelength; psf is m (along T) x n (along D), column-major.
__global__ void k_psf_same(const float *__restrict__ in, float *__restrict__ out,
                           const double *__restrict__ psf, int m, int n, double inv_sum, int D,
                           int T, int ldo) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int d = blockIdx.y, w = blockIdx.z;
    if (t >= T) return;
    const float *s = in + (size_t)w * D * T;
    const int om = m / 2, on = n / 2;
    double acc = 0.0;
    for (int b = 0; b < n; ++b) {
        const int dd = d + on - b;
        if (dd < 0 || dd >= D) continue;
        for (int a = 0; a < m; ++a) {
            const int tt = t + om - a;
            if (tt < 0 || tt >= T) continue;
            acc += psf[a + (size_t)b * m] * (double)s[(size_t)dd * T + tt];
        }
    }
    out[((size_t)w * D + d) * ldo + t] = (float)(acc * inv_sum);
}

// backproject_waveeq.m:35-47: nearest-sample gather into the vector field, the
// products v cos, v sin and their sums as pairs of floats (cos, sin as hi +
// lo in cs[d]).  64 frames of 128 x 128 px, 256 detectors: 2.54 ms (FP64) ->
// 0.48 ms.
__global__ void __launch_bounds__(AN_THREADS) k_bp_gather(
    const float *__restrict__ y, const int32_t *__restrict__ idx,
    const float4 *__restrict__ cs, int nx, int nz, int W, int D, int T, double dtc,
    double *__restrict__ fx, double *__restrict__ fz) {
    const int iz = blockIdx.x * AN_TZ + threadIdx.x % AN_TZ;
    const int ix = blockIdx.y * AN_TX + threadIdx.x / AN_TZ;
    if (ix >= nx || iz >= nz) return;
    const size_t P = (size_t)nx * nz, p = (size_t)ix * nz + iz;
    const int w0 = blockIdx.z * AN_FR;
    const float *s[AN_FR];
#pragma unroll
    for (int f = 0; f < AN_FR; ++f) s[f] = y + (size_t)min(w0 + f, W - 1) * D * T;
    Sum2 ax[AN_FR / 2], az[AN_FR / 2];
#pragma unroll
    for (int f = 0; f < AN_FR / 2; ++f) {
        ax[f].zero();
        az[f].zero();
    }
    const float2 m1 = make_float2(-1.f, -1.f);
#pragma unroll 2
    for (int d = 0; d < D; ++d) {
        const size_t at = (size_t)d * T + __ldg(idx + (size_t)d * P + p);
        const float4 k = __ldg(cs + d);
        const float2 ch = make_float2(k.x, k.x), cl = make_float2(k.y, k.y),
                     sh = make_float2(k.z, k.z), sl = make_float2(k.w, k.w);
#pragma unroll
        for (int f = 0; f < AN_FR / 2; ++f) {
            const float2 v = make_float2(__ldg(s[2 * f] + at), __ldg(s[2 * f + 1] + at));
            const float2 a = __fmul2_rn(v, ch), b = __fmul2_rn(v, sh);
            ax[f].add(a, ffma2(v, cl, ffma2(v, ch, __fmul2_rn(a, m1))));
            az[f].add(b, ffma2(v, sl, ffma2(v, sh, __fmul2_rn(b, m1))));
        }
    }
#pragma unroll
    for (int f = 0; f < AN_FR; ++f) {
        if (w0 + f >= W) break;
        fx[(size_t)(w0 + f) * P + p] = dtc * (f & 1 ? ax[f / 2].y() : ax[f / 2].x());
        fz[(size_t)(w0 + f) * P + p] = dtc * (f & 1 ? az[f / 2].y() : az[f / 2].x());
    }
}

// backproject_waveeq.m:49: fliplr(divergence(fov_x, fov_y, fx, fz)); MATLAB
// gradient: central differences inside, one-sided at the borders.  rx, rz:
// the reciprocal coordinate differences of every column / row.
__global__ void k_div_fliplr(const double *__restrict__ fx, const double *__restrict__ fz,
                             const double *__restrict__ rx, const double *__restrict__ rz,
                             int nx, int nz, float *__restrict__ out) {
    const int P = nx * nz;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int w = blockIdx.y;
    if (p >= P) return;
    const int ix = p / nz, iz = p - ix * nz;
    const double *u = fx + (size_t)w * P, *v = fz + (size_t)w * P;
    const int xa = max(ix - 1, 0), xb = min(ix + 1, nx - 1);
    const int za = max(iz - 1, 0), zb = min(iz + 1, nz - 1);
    const double gx =
        nx > 1 ? (u[(size_t)xb * nz + iz] - u[(size_t)xa * nz + iz]) * rx[ix] : 0.0;
    const double gz =
        nz > 1 ? (v[(size_t)ix * nz + zb] - v[(size_t)ix * nz + za]) * rz[iz] : 0.0;
    out[(size_t)w * P + (size_t)(nx - 1 - ix) * nz + iz] = (float)(gx + gz);
}

// 1 / (difference of the coordinates that k_div_fliplr takes at each place)
static std::vector<double> reciprocal_steps(const double *x, int n) {
    std::vector<double> r(n, 0.0);
    for (int i = 0; i < n && n > 1; ++i)
        r[i] = 1.0 / (x[std::min(i + 1, n - 1)] - x[std::max(i - 1, 0)]);
    return r;
}

// Workspaces of one call, from a stream-ordered pool of the library's own
// (one per device) instead of a dozen cudaMalloc / cudaFree, which synchronise, per
// call.  The pool keeps at most POOL_KEEP bytes between calls, the rest goes
// back at the call's synchronisation; msot_release_workspaces gives back what it keeps.
constexpr uint64_t POOL_KEEP = 512ull << 20;
constexpr int POOL_DEVICES = 64;
static cudaMemPool_t g_pools[POOL_DEVICES] = {};
static std::mutex g_pools_mu;
static cudaMemPool_t analytic_pool() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= POOL_DEVICES) return nullptr;
    std::lock_guard<std::mutex> g(g_pools_mu);
    if (!g_pools[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
        uint64_t keep = POOL_KEEP;
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        g_pools[dev] = p;
    }
    return g_pools[dev];
}

// Host tables are copied asynchronously and, where the GPU reads pageable memory
// itself, without a staging copy: they live here until the copies are done.
struct DevMem {
    cudaStream_t st;
    std::vector<void *> ptrs;
    std::vector<std::vector<char>> host;
    explicit DevMem(cudaStream_t s) : st(s) {}
    DevMem(const DevMem &) = delete;
    DevMem &operator=(const DevMem &) = delete;
    ~DevMem() {
        if (!host.empty()) cudaStreamSynchronize(st);
        for (void *p : ptrs) cudaFreeAsync(p, st);
    }
    template <class T>
    int get(T **p, size_t n) {
        void *q = nullptr;
        cudaMemPool_t pool = analytic_pool();
        if (!pool || cudaMallocFromPoolAsync(&q, n * sizeof(T), pool, st) != cudaSuccess) {
            cudaGetLastError();  // reported here, not by the next launch check
            set_error("analytic: allocation of %zu bytes failed", n * sizeof(T));
            return MSOT_ENOMEM;
        }
        ptrs.push_back(q);
        *p = static_cast<T *>(q);
        return MSOT_OK;
    }
    template <class T>
    int put(T **p, const T *h, size_t n) {
        int rc = get(p, n);
        if (rc) return rc;
        const char *b = reinterpret_cast<const char *>(h);
        host.emplace_back(b, b + n * sizeof(T));
        MSOT_CUDA_TRY(
            cudaMemcpyAsync(*p, host.back().data(), n * sizeof(T), cudaMemcpyHostToDevice, st));
        return MSOT_OK;
    }
};

#define RC(x)                                                                              \
    do {                                                                                   \
        int rc_ = (x);                                                                     \
        if (rc_) return rc_;                                                               \
    } while (0)

// Shared set-up: detector angles (dmas_cf.m:45-46) and the index table.
static int index_table(DevMem &m, int D, int T, const double *x, int nx, const double *z, int nz,
                       double c, double fs, double n_crop, double coverage, double R,
                       cudaStream_t st, int32_t **d_idx, float4 **d_cs) {
    std::vector<double> ca(D), sa(D);
    const double off = (180.0 - coverage) / 2.0, step = D > 1 ? coverage / (D - 1) : 0.0;
    const double pi = 3.141592653589793238462643383279502884;
    for (int d = 0; d < D; ++d) {
        const double a = -(off + step * d) * pi / 180.0;
        ca[d] = std::cos(a);
        sa[d] = std::sin(a);
    }
    std::vector<float4> cs(D);  // hi and lo parts for k_bp_gather
    for (int d = 0; d < D; ++d) {
        const float ch = (float)ca[d], sh = (float)sa[d];
        cs[d] = make_float4(ch, (float)(ca[d] - (double)ch), sh, (float)(sa[d] - (double)sh));
    }
    std::vector<float> xf(x, x + nx), zf(z, z + nz);
    std::vector<float2> det(D);
    for (int d = 0; d < D; ++d) det[d] = make_float2((float)(ca[d] * R), (float)(sa[d] * R));
    float *dxf, *dzf;
    float2 *ddet;
    RC(m.put(&dxf, xf.data(), nx));
    RC(m.put(&dzf, zf.data(), nz));
    RC(m.put(&ddet, det.data(), D));
    double *dx, *dz, *dc, *ds;
    int *derr;
    RC(m.put(&dc, ca.data(), D));
    RC(m.put(&ds, sa.data(), D));
    RC(m.put(d_cs, cs.data(), D));
    RC(m.put(&dx, x, nx));
    RC(m.put(&dz, z, nz));
    RC(m.get(d_idx, (size_t)D * nx * nz));
    RC(m.get(&derr, 1));
    MSOT_CUDA_TRY(cudaMemsetAsync(derr, 0, sizeof(int), st));
    const int P = nx * nz;
    // FP32 estimate: coordinates, their difference, the distance and the
    // offset carry below eight roundings of 2^-24 of `reach` samples together
    double far = std::fabs(R);
    for (int i = 0; i < nx; ++i) far = std::max(far, std::fabs(x[i]));
    for (int i = 0; i < nz; ++i) far = std::max(far, std::fabs(z[i]));
    const double reach = 4.0 * far * std::fabs(fs / c) + std::fabs(n_crop) + 2.0;
    const float tol = (float)std::min(0.5, 8.0 * std::ldexp(reach, -24));
    KLAUNCH(k_nearest_index<<<dim3(div_up(P, 256), D), 256, 0, st>>>(
        dc, ds, dx, dz, dxf, dzf, ddet, (float)(fs / c), (float)(-n_crop), nx, nz, D, R, c, fs, (1.0 + n_crop) / fs, T, tol, *d_idx, derr));
    MSOT_LAUNCH_CHECK();
    int herr = 0;
    MSOT_CUDA_TRY(cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, st));
    MSOT_CUDA_TRY(cudaStreamSynchronize(st));
    if (herr) {
        set_error("nearest-sample index outside the sinogram (the reference errors here)");
        return MSOT_ERANGE;
    }
    return MSOT_OK;
}

}  // namespace msot

using namespace msot;

extern "C" {

int msot_release_workspaces(void) {
    std::lock_guard<std::mutex> g(g_pools_mu);
    for (int dev = 0; dev < POOL_DEVICES; ++dev) {
        if (!g_pools[dev]) continue;
        int was = 0;
        MSOT_CUDA_TRY(cudaGetDevice(&was));
        MSOT_CUDA_TRY(cudaSetDevice(dev));
        cudaError_t e = cudaDeviceSynchronize();  // frees of calls just made
        if (e == cudaSuccess) e = cudaMemPoolTrimTo(g_pools[dev], 0);
        cudaSetDevice(was);
        MSOT_CUDA_TRY(e);
    }
    return MSOT_OK;
}

int msot_dmas_cf(const float *d_sig, int W, int D, int T, const double *x, int nx,
                 const double *z, int nz, double c, double fs, double n_crop, double coverage_deg,
                 double radius, float *d_dmas_cf, float *d_dmas, float *d_cf, float *d_das,
                 void *stream) {
    if (!d_sig || !x || !z || !d_dmas_cf || !d_dmas || !d_cf || !d_das || W <= 0 || D <= 1 ||
        T <= 0 || nx <= 0 || nz <= 0) {
        set_error("dmas_cf: bad arguments");
        return MSOT_EINVAL;
    }
    cudaStream_t st = (cudaStream_t)stream;
    DevMem m(st);
    int32_t *idx;
    float4 *cs;
    RC(index_table(m, D, T, x, nx, z, nz, c, fs, n_crop, coverage_deg, radius, st, &idx, &cs));
    unsigned int *mx;
    RC(m.get(&mx, 1));
    MSOT_CUDA_TRY(cudaMemsetAsync(mx, 0, sizeof(unsigned int), st));
    const size_t n = (size_t)W * D * T;
    KLAUNCH(k_max_abs<<<1024, 256, 0, st>>>(d_sig, n, mx));
    const dim3 grid(div_up(nz, AN_TZ), div_up(nx, AN_TX), div_up(W, AN_FR));
    KLAUNCH(k_dmas_cf<<<grid, AN_THREADS, 0, st>>>(d_sig, idx, mx, nx, nz, W, D, T, d_dmas_cf,
                                                   d_dmas, d_cf, d_das));
    MSOT_LAUNCH_CHECK();
    MSOT_CUDA_TRY(cudaStreamSynchronize(st));
    return MSOT_OK;
}

int msot_backproject_waveeq(const float *d_sig, int W, int D, int T, const double *x, int nx,
                            const double *z, int nz, double c, double fs, double n_crop,
                            double coverage_deg, double radius, const double *psf, int psf_m,
                            int psf_n, const float *d_K, int K_n, float *d_out, void *stream) {
    if (!d_sig || !x || !z || !psf || !d_K || !d_out || W <= 0 || D <= 1 || T <= 1 || nx <= 0 ||
        nz <= 0 || psf_m <= 0 || psf_n <= 0) {
        set_error("backproject_waveeq: bad arguments");
        return MSOT_EINVAL;
    }
    const long crop = std::lround(n_crop);
    if ((double)crop != n_crop || crop < 0 || crop + T > K_n) {
        set_error("backproject_waveeq: K (%d x %d) does not cover samples %ld..%ld", K_n, K_n,
                  crop + 1, crop + T);
        return MSOT_EINVAL;
    }
    double psum = 0.0;
    for (int i = 0; i < psf_m * psf_n; ++i) psum += psf[i];
    if (psum == 0.0) {
        set_error("backproject_waveeq: psf sums to zero");
        return MSOT_EINVAL;
    }
    cudaStream_t st = (cudaStream_t)stream;
    DevMem m(st);
    int32_t *idx;
    float4 *cs;
    double *dpsf, *fx, *fz, *drx, *drz;
    RC(index_table(m, D, T, x, nx, z, nz, c, fs, n_crop, coverage_deg, radius, st, &idx, &cs));
    RC(m.put(&drx, reciprocal_steps(x, nx).data(), nx));
    RC(m.put(&drz, reciprocal_steps(z, nz).data(), nz));
    float *s1, *s2;
    const size_t n = (size_t)W * D * T;
    const int P = nx * nz;
    const int ld = (T + 3) / 4 * 4;  // the GEMM's operand: 16-byte aligned columns
    RC(m.get(&s1, n));
    RC(m.get(&s2, (size_t)W * D * ld));
    RC(m.get(&fx, (size_t)W * P));
    RC(m.get(&fz, (size_t)W * P));
    const double dt = 1.0 / fs;
    std::vector<float2> fac(T);
    for (int t = 0; t < T; ++t) {
        const double f = 0.5 / (c * (t + 1 + n_crop));
        const float h = (float)f;
        fac[t] = make_float2(h, (float)(f - (double)h));
    }
    float2 *dfac;
    RC(m.put(&dfac, fac.data(), T));
    // a 1 x 1 psf divided by its own sum is the identity
    const bool one = psf_m == 1 && psf_n == 1 && std::isfinite(psf[0]);
    size_t ct_smem = (size_t)CT_WARPS * 32 * (((T + 31) / 32) | 1) * sizeof(float);
    const int staged = ct_smem <= 200 * 1024;
    if (!staged) ct_smem = 0;
    RC(set_smem(k_cumtrapz, ct_smem));
    KLAUNCH(k_cumtrapz<<<div_up(W * D, CT_WARPS), 32 * CT_WARPS, ct_smem, st>>>(
        d_sig, one ? s2 : s1, W * D, T, one ? ld : T, staged, dfac));
    if (!one) {
        RC(m.put(&dpsf, psf, (size_t)psf_m * psf_n));
        KLAUNCH(k_psf_same<<<dim3(div_up(T, 128), D, W), 128, 0, st>>>(s1, s2, dpsf, psf_m, psf_n,
                                                                     1.0 / psum, D, T, ld));
    }
    MSOT_LAUNCH_CHECK();
    // s1 = K(acq, acq) * s2 * dt : one column-major GEMM over all (d, w)
    // columns, on the tensor cores (gemm_tc.cu)
    const float *Ksub = d_K + (size_t)crop * K_n + crop;
    RC(tc_sgemm(T, D * W, T, (float)dt, Ksub, K_n, s2, ld, s1, T, st));
    const dim3 grid(div_up(nz, AN_TZ), div_up(nx, AN_TX), div_up(W, AN_FR));
    KLAUNCH(k_bp_gather<<<grid, AN_THREADS, 0, st>>>(s1, idx, cs, nx, nz, W, D, T, dt * c, fx, fz));
    KLAUNCH(k_div_fliplr<<<dim3(div_up(P, 256), W), 256, 0, st>>>(fx, fz, drx, drz, nx, nz, d_out));
    MSOT_LAUNCH_CHECK();
    MSOT_CUDA_TRY(cudaStreamSynchronize(st));
    return tc_sgemm_check();
}

}  // extern "C"

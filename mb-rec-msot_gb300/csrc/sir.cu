// sir.cu -- the interpolation with spatial impulse responses, forward
// (forwardMex.cpp:118-160) and adjoint (transposeMex.cpp:115-158).
//
// A (pixel, detector) pair deposits its SIR column h convolved with its tri
// taps.  For tau = b + f the tri weights are linear in f on the three pieces
// between their kinks (operator.cu, bucket decomposition), so the composite is
// e[m] = A[m] + f B[m] with one table row (A, B) per column and piece, built
// once per plan: one 8-byte load and one FMA per tap, shared by all instances,
// instead of 2r + 2 FMAs.
//
//   k_sir_fwd2  CTA = (64 output samples, detector, NI instances): lanes hold
//               two samples each and walk the pairs whose window reaches the
//               tile (sorted by window start), accumulating in registers; four
//               warps share the list and are summed at the end.  No atomics:
//               deterministic, where the column in shared memory took one
//               atomic (a compare-and-swap loop for FP32) per tap and instance.
//   k_sir_adj2  half warp = two pixels: lanes over the window's taps, per detector
//               one e[m] for all instances against the block's samples in
//               shared memory, the taps added before the next detector's.
//
// 128 x 128 px, 256 x 2030 samples, 8 instances, columns of 31 samples on
// average: forward 2398 -> 590 us, adjoint 1187 -> 740 us.  Bound:
// issue slots (address and window arithmetic per pair, one packed FMA per tap
// and two instances) and the table rows' L1 lines.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "ptx.cuh"

namespace msot {

constexpr int SF_T = 64, SF_WARPS = 4;      // forward: samples per CTA, warps sharing a list
// chains of a sample's sum in each warp: a few hundred terms cancel to a tenth of them,
// and one chain was less exact than the former kernel's atomics (128 x 128 px, one
// image: 3.1e-6 of A x, there 2.2e-6, now 2.0e-6; 8 images 550 -> 624 us)
constexpr int SF_CH = 2;
constexpr int SA_THREADS = 256, SA_PIX = 32;  // adjoint: pixels per CTA, two per half warp

// (A, B)[m] of every (column, piece), m = j + F + k over tri taps j = -F ..
// F + 1 and column samples k; row length S + 2F + 1
__global__ void __launch_bounds__(128) k_sir_table(const float *__restrict__ sir,
                                                   const int2 *__restrict__ se, int S, int F,
                                                   double r, float2 *__restrict__ tab) {
    const int row = blockIdx.x, s = row / 3, piece = row % 3, RL = S + 2 * F + 1;
    const double ir = 1.0 / r;
    const double a = r - F, b = F + 1 - r;  // kinks: e1 ends at a, e2 starts at b
    const bool has1 = piece == 0 || (piece == 1 && a > b);
    const bool has2 = piece == 2 || (piece == 1 && a > b);
    const int2 e = se[s];
    for (int m = threadIdx.x; m < RL; m += blockDim.x) {
        double va = 0.0, vb = 0.0;
        for (int j = -F; j <= F + 1; ++j) {
            const int k = m - F - j;
            if (k < e.x || k > e.y) continue;
            double wa, wb;  // weight of tap j = wa + wb f
            if (j == -F) {
                wa = has1 ? a * ir : 0.0;
                wb = has1 ? -ir : 0.0;
            } else if (j == F + 1) {
                wa = has2 ? -b * ir : 0.0;
                wb = has2 ? ir : 0.0;
            } else {
                wa = 1.0 - abs(j) * ir;
                wb = j <= 0 ? -ir : ir;
            }
            const double h = sir[(size_t)s * S + k];
            va += wa * h;
            vb += wb * h;
        }
        tab[(size_t)row * RL + m] = make_float2((float)va, (float)vb);
    }
}

// Every load of the two kernels has an address inside its array, also where the
// value is not used: no load depends on a predicate for that (windows reach far
// past both ends of a row's table and of the sinogram).  A precaution: an earlier
// form, which predicated these loads instead, met a memory fault, and reading
// its entries, rows, offsets and indices did not show why (a load that is
// predicated off reads nothing).

// window start (low 16 bits hold the length)
__device__ __forceinline__ int se_start(int v) { return v >> 16; }
__device__ __forceinline__ int se_len(int v) { return v & 0xffff; }

template <int NI>
__global__ void __launch_bounds__(32 * SF_WARPS) k_sir_fwd2(
    const int4 *__restrict__ ent, const int32_t *__restrict__ off, int jmin, int nj, int maxlen,
    const float2 *__restrict__ tab, const float *__restrict__ xpm, float *__restrict__ raw, int P,
    int D, int T, int W, float scale) {
    constexpr int NP = (NI + 1) / 2;  // instance pairs
    __shared__ float red[SF_WARPS - 1][NI][SF_T];
    const int d = blockIdx.y, w0 = blockIdx.z * NI, t0 = blockIdx.x * SF_T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // samples t0 + lane and t0 + 32 + lane, SF_CH chains each
    float2 part[SF_CH][2][NP];
#pragma unroll
    for (int i = 0; i < SF_CH * 2 * NP; ++i)
        part[i / (2 * NP)][i / NP % 2][i % NP] = make_float2(0.f, 0.f);
    // pairs whose window starts in (t0 - maxlen, t0 + 64)
    const int32_t *o = off + (size_t)d * (nj + 1);
    const int ja = min(max(t0 - maxlen + 1 - jmin, 0), nj), jb = min(max(t0 + SF_T - jmin, 0), nj);
    const int n0 = __ldg(o + ja), n1 = __ldg(o + jb);
    const int4 *e = ent + (size_t)d * P;
    const float *x = xpm + (size_t)blockIdx.z * P * NI;
    constexpr int U = 4;  // pairs in flight; the next ones' entries load meanwhile
    int4 qn[U];
    auto fetch = [&](int j) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            qn[u] = __ldg(e + min(j + u, P - 1));
            if (j + u >= n1) qn[u].y &= (int)0xffff0000;  // length 0
        }
    };
    fetch(n0 + warp * U);
    for (int j = n0 + warp * U; j < n1; j += SF_WARPS * U) {
        int4 q[U];
        float2 xv[U][NP];
#pragma unroll
        for (int u = 0; u < U; ++u) q[u] = qn[u];
        fetch(j + SF_WARPS * U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float *xp = x + (size_t)q[u].w * NI;
            if constexpr (NI % 4 == 0) {
#pragma unroll
                for (int i = 0; i < NP; i += 2) {
                    const float4 v = __ldg(reinterpret_cast<const float4 *>(xp + 2 * i));
                    xv[u][i] = make_float2(v.x, v.y);
                    xv[u][i + 1] = make_float2(v.z, v.w);
                }
            } else {
                xv[u][0] = make_float2(__ldg(xp), NI > 1 ? __ldg(xp + NI - 1) : 0.f);
            }
        }
        float2 a[U][2];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int m = t0 + lane - se_start(q[u].y), last = max(se_len(q[u].y) - 1, 0);
            const float2 *row = tab + q[u].x;
            a[u][0] = __ldg(row + min(max(m, 0), last));
            a[u][1] = __ldg(row + min(max(m + 32, 0), last));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float f = __int_as_float(q[u].z);
            const unsigned m = (unsigned)(t0 + lane - se_start(q[u].y)), len = se_len(q[u].y);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float ev = fmaf(f, a[u][h].y, a[u][h].x);
                const float2 e2 = make_float2(ev, ev);
                if (m + 32u * h < len) {  // a NaN pixel reaches its own window only
#pragma unroll
                    for (int i = 0; i < NP; ++i)
                        part[u % SF_CH][h][i] = ffma2(e2, xv[u][i], part[u % SF_CH][h][i]);
                }
            }
        }
    }
    float2 acc[2][NP];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            acc[h][i] = part[0][h][i];
#pragma unroll
            for (int c = 1; c < SF_CH; ++c) acc[h][i] = fadd2(acc[h][i], part[c][h][i]);
        }
#pragma unroll
    for (int i = 0; i < NI && warp > 0; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            red[warp - 1][i][32 * h + lane] = i & 1 ? acc[h][i / 2].y : acc[h][i / 2].x;
    __syncthreads();
    if (warp > 0) return;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        if (w0 + i >= W) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v = i & 1 ? acc[h][i / 2].y : acc[h][i / 2].x;
#pragma unroll
            for (int k = 0; k < SF_WARPS - 1; ++k) v += red[k][i][32 * h + lane];
            const int t = t0 + 32 * h + lane;
            if (t < T) raw[((size_t)(w0 + i) * D + d) * T + t] = v * scale;
        }
    }
}

// CTA = (SA_PIX pixels, NI instances).  Per detector the samples that the
// block's windows span (aspan) lie in shared memory, [sample][instance]; a
// half warp takes two pixels, lanes over taps, the next detector's samples are
// loaded into registers meanwhile.
//
// A detector's taps are added to one value before they enter the pixel's sum.
// The composite row is smooth and the recordings oscillate, so taps cancel within
// one detector and not tap by tap over the detectors: lanes that each kept a
// tap's sum over all detectors lost a factor of 4 at 80 x 80 px and of 40 at 60 x
// 60.  The half warp reduces and scatters: lane bits 3, 2, 1, 0 take the pixel, the
// group of four instances and the instance in it, and each lane ends with one
// (pixel, instance).  Pixels and groups sit in the lanes' registers in the order
// that lets a lane send its second half as it is; no selection there.
template <int NI>
__global__ void __launch_bounds__(SA_THREADS) k_sir_adj2(
    const int4 *__restrict__ ent, const int2 *__restrict__ aspan, const float2 *__restrict__ tab,
    const float *__restrict__ raw, float *__restrict__ out, int P, int D, int T, int W,
    int span_max, int det_per_group, size_t part_stride) {
    constexpr int QN = NI / 4;                       // 16-byte groups per sample
    constexpr int PPH = SA_PIX / (SA_THREADS / 16);  // pixels per half warp
    static_assert(PPH == 2 && (NI == 4 || NI == 8), "lane bits of the reduction");
    constexpr int NPRE = 3;                          // groups in flight per thread
    extern __shared__ float4 ys[];  // [2][QN][span_max]
    const int l = threadIdx.x & 15, half = threadIdx.x >> 4;
    const int b3 = l >> 3, b2 = l >> 2 & 1, b1 = l >> 1 & 1, b0 = l & 1;
    const int blk = blockIdx.x, w0 = blockIdx.y * NI;
    const int4 *e = ent + (size_t)blk * D * SA_PIX;
    const size_t DT = (size_t)D * T;
    // slot k of a lane holds pixel k ^ b3 of its half warp, slot g (NI = 8) the
    // instances 4 (g ^ b2) ..
    const int pix[PPH] = {b3 * (SA_THREADS / 16) + half, (b3 ^ 1) * (SA_THREADS / 16) + half};
    float sum = 0.f;
    float4 pre[NPRE];
    // group g of the staging: sample g / QN, instances 4 (g % QN) ..; zero outside
    // the row, instances past W repeat the last one and are not stored
    auto load = [&](int d, int g, int2 sp) {
        const int k = g / QN, tt = sp.x + k, i0 = w0 + 4 * (g % QN);
        const bool ok = k < sp.y - sp.x && tt >= 0 && tt < T;
        const float *y = raw + (size_t)d * T + min(max(tt, 0), T - 1);
        float4 v;
        v.x = __ldg(y + (size_t)min(i0, W - 1) * DT);
        v.y = __ldg(y + (size_t)min(i0 + 1, W - 1) * DT);
        v.z = __ldg(y + (size_t)min(i0 + 2, W - 1) * DT);
        v.w = __ldg(y + (size_t)min(i0 + 3, W - 1) * DT);
        return ok ? v : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto slot = [&](int buf, int g) {
        return ys + ((size_t)buf * QN + g % QN) * span_max + g / QN;
    };
    const int d0 = blockIdx.z * det_per_group, d1 = min(D, d0 + det_per_group);
    int4 qn[PPH];  // the next detector's pairs
    {
        const int2 sp = __ldg(aspan + (size_t)blk * D + d0);
        for (int g = threadIdx.x; g < QN * (sp.y - sp.x); g += SA_THREADS)
            *slot(0, g) = load(d0, g, sp);
#pragma unroll
        for (int k = 0; k < PPH; ++k)
            qn[k] = __ldg(e + (size_t)d0 * SA_PIX + pix[k]);
    }
    for (int d = d0; d < d1; ++d) {
        const int buf = (d - d0) & 1;
        const int2 sp = __ldg(aspan + (size_t)blk * D + d);
        int2 sn = make_int2(0, 0);
        __syncthreads();  // buffer `buf` is complete, the other one is free
        if (d + 1 < d1) {
            sn = __ldg(aspan + (size_t)blk * D + d + 1);
#pragma unroll
            for (int k = 0; k < NPRE; ++k)
                if (threadIdx.x + k * SA_THREADS < QN * (sn.y - sn.x))
                    pre[k] = load(d + 1, threadIdx.x + k * SA_THREADS, sn);
        }
        const float4 *y = ys + (size_t)buf * QN * span_max;
        int4 qc[PPH];
        float2 tv[PPH][3];  // the first 48 taps' rows
#pragma unroll
        for (int k = 0; k < PPH; ++k) {
            qc[k] = qn[k];
            const int last = max(se_len(qc[k].y) - 1, 0);
#pragma unroll
            for (int h = 0; h < 3; ++h) tv[k][h] = __ldg(tab + qc[k].x + min(16 * h + l, last));
            qn[k] = __ldg(e + (size_t)min(d + 1, D - 1) * SA_PIX + pix[k]);
        }
        float2 acc[PPH][NI / 2];
#pragma unroll
        for (int k = 0; k < PPH; ++k)
#pragma unroll
            for (int i = 0; i < NI / 2; ++i) acc[k][i] = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < PPH; ++k) {
            const int4 q = qc[k];
            const int len = se_len(q.y), last = max(len - 1, 0);
            const int at = se_start(q.y) - sp.x;  // window start within the span
            const float f = __int_as_float(q.z);
            for (int c = 0; c < len; c += 48) {
                if (c)
#pragma unroll
                    for (int h = 0; h < 3; ++h)
                        tv[k][h] = __ldg(tab + q.x + min(c + 16 * h + l, last));
#pragma unroll
                for (int h = 0; h < 3; ++h) {
                    const int m = c + 16 * h + l;
                    const float ev = fmaf(f, tv[k][h].y, tv[k][h].x);
                    const float2 e2 = make_float2(ev, ev);
                    const int s = min(max(at + min(m, last), 0), span_max - 1);
#pragma unroll
                    for (int g = 0; g < QN; ++g) {
                        const float4 v = y[(QN == 2 ? g ^ b2 : g) * span_max + s];
                        if (m < len) {
                            acc[k][2 * g] = ffma2(e2, make_float2(v.x, v.y), acc[k][2 * g]);
                            acc[k][2 * g + 1] = ffma2(e2, make_float2(v.z, v.w), acc[k][2 * g + 1]);
                        }
                    }
                }
            }
        }
        // taps of this detector: the other lanes' parts of what this lane keeps
        float2 v[NI / 2];
#pragma unroll
        for (int i = 0; i < NI / 2; ++i) {
            v[i].x = acc[0][i].x + __shfl_xor_sync(0xffffffffu, acc[1][i].x, 8);
            v[i].y = acc[0][i].y + __shfl_xor_sync(0xffffffffu, acc[1][i].y, 8);
        }
        if constexpr (NI == 8) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                v[i].x += __shfl_xor_sync(0xffffffffu, v[2 + i].x, 4);
                v[i].y += __shfl_xor_sync(0xffffffffu, v[2 + i].y, 4);
            }
        }
        const int hi = NI == 8 ? b1 : b2, lo = NI == 8 ? b0 : b1;
        float2 u = hi ? v[1] : v[0];
        const float2 o = hi ? v[0] : v[1];
        u.x += __shfl_xor_sync(0xffffffffu, o.x, NI == 8 ? 2 : 4);
        u.y += __shfl_xor_sync(0xffffffffu, o.y, NI == 8 ? 2 : 4);
        float t = (lo ? u.y : u.x) + __shfl_xor_sync(0xffffffffu, lo ? u.x : u.y, NI == 8 ? 1 : 2);
        if constexpr (NI == 4) t += __shfl_xor_sync(0xffffffffu, t, 1);
        sum += t;
        if (d + 1 < d1) {
            const int n = QN * (sn.y - sn.x);
#pragma unroll
            for (int k = 0; k < NPRE; ++k)
                if (threadIdx.x + k * SA_THREADS < n)
                    *slot(buf ^ 1, threadIdx.x + k * SA_THREADS) = pre[k];
            for (int g = threadIdx.x + NPRE * SA_THREADS; g < n; g += SA_THREADS)
                *slot(buf ^ 1, g) = load(d + 1, g, sn);
        }
    }
    const int p = blk * SA_PIX + pix[0], i = NI == 8 ? 4 * b2 + 2 * b1 + b0 : 2 * b2 + b1;
    if ((NI == 8 || !b0) && p < P && w0 + i < W)
        out[blockIdx.z * part_stride + (size_t)(w0 + i) * P + p] = sum;
}

// Tables of the two kernels from the travel times tfx [D][P], the 0-based
// inclusive column spans and the columns sidx [D][P] (1-based).  Leaves
// p.sir_tab null (the kernels of operator.cu serve the plan) when the packed
// fields or the table would not fit.
int sir_build(Plan &p, const int32_t *tfx, const int32_t *sidx, const std::vector<int2> &se,
              size_t &bytes) {
    const int F = p.F, RL = p.S + 2 * F + 1, half = p.S / 2;
    const size_t tab = (size_t)p.NS * 3 * RL;
    if (p.T > 30000 || RL > 2000 || tab > (size_t)INT32_MAX / 2) return MSOT_OK;
    for (const int2 &e : se)
        if (e.y < e.x) return MSOT_OK;
    const double a = p.radius - F, b = F + 1 - p.radius;
    const float p1 = (float)std::min(a, b), p2 = (float)std::max(a, b);
    const int mask = (1 << p.frac_bits) - 1;
    const float step = std::ldexp(1.f, -p.frac_bits);
    // window starts: b - half - F + first column sample
    auto start = [&](int32_t tau, int s) { return (tau >> p.frac_bits) - half - F + se[s].x; };
    const size_t PD = (size_t)p.P * p.D;
    int jmin = INT_MAX, jmax = INT_MIN, maxlen = 0;
    double sum = 0.0;
    for (size_t i = 0; i < PD; ++i) {
        const int s = sidx[i] - 1, j = start(tfx[i], s);
        jmin = std::min(jmin, j);
        jmax = std::max(jmax, j);
        maxlen = std::max(maxlen, se[s].y - se[s].x + 2 * F + 2);
        sum += se[s].y - se[s].x + 1;
    }
    p.sir_len_mean = sum / (double)PD;
    if (jmin < -32000 || jmax > 32000) return MSOT_OK;
    const int nj = jmax - jmin + 1;
    auto entry = [&](int32_t tau, int s, int pix) {
        const float f = (float)(tau & mask) * step;
        const int piece = (f >= p1) + (f >= p2);
        const int len = se[s].y - se[s].x + 2 * F + 2;
        int4 q;
        q.x = (3 * s + piece) * RL + se[s].x;
        q.y = (int)((uint32_t)start(tau, s) << 16 | (uint32_t)len);
        std::memcpy(&q.z, &f, sizeof f);
        q.w = pix;
        return q;
    };
    const int blocks = div_up(p.P, SA_PIX);
    const size_t na = (size_t)blocks * p.D * SA_PIX;
    std::vector<int32_t> off((size_t)p.D * (nj + 1), 0);
    std::vector<int4> fe(PD), ae(na, make_int4(0, 0, 0, 0));
    std::vector<int2> asp((size_t)blocks * p.D, make_int2(INT_MAX, INT_MIN));
    for (int d = 0; d < p.D; ++d) {
        const int32_t *tf = tfx + (size_t)d * p.P, *si = sidx + (size_t)d * p.P;
        int32_t *o = off.data() + (size_t)d * (nj + 1);
        for (int q = 0; q < p.P; ++q) {
            const int s = si[q] - 1, j = start(tf[q], s);
            ++o[j - jmin + 1];
        }
        for (int j = 0; j < nj; ++j) o[j + 1] += o[j];
        std::vector<int32_t> fill(o, o + nj);
        for (int q = 0; q < p.P; ++q) {
            const int4 v = entry(tf[q], si[q] - 1, q);
            fe[(size_t)d * p.P + fill[(v.y >> 16) - jmin]++] = v;
            ae[((size_t)(q / SA_PIX) * p.D + d) * SA_PIX + q % SA_PIX] = v;
            int2 &sp = asp[(size_t)(q / SA_PIX) * p.D + d];
            sp.x = std::min(sp.x, v.y >> 16);
            sp.y = std::max(sp.y, (v.y >> 16) + (v.y & 0xffff));
        }
    }
    int span = 1;
    for (const int2 &v : asp) span = std::max(span, v.y - v.x);
    span = (span + 7) / 8 * 8;  // lanes of two groups of instances meet other banks
    if ((size_t)span * 2 * 32 > 100 * 1024) return MSOT_OK;  // two buffers of 8 instances
    p.sir_span_max = span;
    MSOT_MALLOC_TRY(cudaMalloc(&p.sir_aspan, asp.size() * sizeof(int2)));
    MSOT_CUDA_TRY(cudaMemcpy(p.sir_aspan, asp.data(), asp.size() * sizeof(int2),
                             cudaMemcpyHostToDevice));
    MSOT_MALLOC_TRY(cudaMalloc(&p.sir_fent, PD * sizeof(int4)));
    MSOT_MALLOC_TRY(cudaMalloc(&p.sir_aent, na * sizeof(int4)));
    MSOT_MALLOC_TRY(cudaMalloc(&p.sir_off, off.size() * sizeof(int32_t)));
    MSOT_CUDA_TRY(cudaMemcpy(p.sir_fent, fe.data(), PD * sizeof(int4), cudaMemcpyHostToDevice));
    MSOT_CUDA_TRY(cudaMemcpy(p.sir_aent, ae.data(), na * sizeof(int4), cudaMemcpyHostToDevice));
    MSOT_CUDA_TRY(cudaMemcpy(p.sir_off, off.data(), off.size() * sizeof(int32_t),
                             cudaMemcpyHostToDevice));
    MSOT_MALLOC_TRY(cudaMalloc(&p.sir_tab, tab * sizeof(float2)));
    bytes += (PD + na) * sizeof(int4) + asp.size() * sizeof(int2) + off.size() * sizeof(int32_t) + tab * sizeof(float2);
    p.sir_jmin = jmin;
    p.sir_nj = nj;
    p.sir_maxlen = maxlen;
    return MSOT_OK;
}

// after the columns are on the device
int sir_build_table(Plan &p) {
    KLAUNCH(k_sir_table<<<3 * p.NS, 128>>>(p.sir, p.sir_se, p.S, p.F, p.radius, p.sir_tab));
    MSOT_LAUNCH_CHECK();
    return MSOT_OK;
}

int launch_sir_forward2(const Plan &pl, const float *xpm, float *raw, int W, int wt, float scale,
                        cudaStream_t st) {
    const dim3 grid(div_up(pl.T, SF_T), pl.D, div_up(W, wt));
#define SIRF(NI)                                                                           \
    KLAUNCH(k_sir_fwd2<NI><<<grid, 32 * SF_WARPS, 0, st>>>(                                \
        pl.sir_fent, pl.sir_off, pl.sir_jmin, pl.sir_nj, pl.sir_maxlen, pl.sir_tab, xpm, raw, \
        pl.P, pl.D, pl.T, W, scale))
    if (wt == 8) SIRF(8);
    else if (wt == 4) SIRF(4);
    else if (wt == 2) SIRF(2);
    else SIRF(1);
#undef SIRF
    MSOT_LAUNCH_CHECK();
    return MSOT_OK;
}

int launch_sir_adjoint2(const Plan &pl, const float *raw, float *x, int W, float scale,
                        cudaStream_t st) {
    const int ni = W >= 5 ? 8 : 4;
    // detector groups (partial images, summed in order) until the CTAs fill
    // whole waves of three per SM
    const int base = div_up(pl.P, SA_PIX) * div_up(W, ni), slots = 3 * sm_count();
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
    const dim3 grid(div_up(pl.P, SA_PIX), div_up(W, ni), groups);
    const size_t smem = (size_t)2 * (ni / 4) * pl.sir_span_max * sizeof(float4);
    int rc;
#define SIRA(NI)                                                                           \
    do {                                                                                   \
        if ((rc = set_smem(k_sir_adj2<NI>, smem)) != MSOT_OK) return rc;                   \
        KLAUNCH(k_sir_adj2<NI><<<grid, SA_THREADS, smem, st>>>(                            \
            pl.sir_aent, pl.sir_aspan, pl.sir_tab, raw, pl.scr_part, pl.P, pl.D, pl.T, W,  \
            pl.sir_span_max, dpg, stride));                                                \
    } while (0)
    if (ni == 8) SIRA(8);
    else SIRA(4);
#undef SIRA
    MSOT_LAUNCH_CHECK();
    return sum_parts(pl.scr_part, x, stride, groups, scale, st);
}

}  // namespace msot

// gemm_tc.cu -- FP32-accurate GEMM on the sm_103a tensor cores:
//   C (M x N) = alpha * A (M x K) * B (K x N), all column-major FP32.
// Used for the dense products of backproject_waveeq.m:33 (K(t, t') times the
// radial integrals) and of the pre-processing's zero-phase filter (the T x T
// circulant of ifft(|H|^2), filter_butter_zero_phase.m:42-48).
//
// Precision: each operand is split into a TF32 head and a TF32 tail
// (x = hi + lo, hi = tf32(x), lo = tf32(x - hi)) and the product is
// hi*hi + hi*lo + lo*hi, three tcgen05.mma kind::tf32 per K step with FP32
// accumulation in TMEM: about 2^-21 relative per product, the order of a
// plain FP32 GEMM.
//
// CTA = one 128 x NT tile of C (NT = 256, 128 or 64), accumulator in TMEM,
// warp-specialised: eight producer warps load the raw FP32 panels of a K stage
// of 32 into registers (one stage ahead), split them and store the four panels
// (A hi / lo, B hi / lo) in shared memory in the canonical K-major, no-swizzle
// layout (8-row x 16-byte core matrices, K groups of 4 side by side); one
// thread of a ninth warp issues the 12 MMAs of a stage and commits them to the
// buffer's "empty" mbarrier.  The split stays inside the SM: packed operands
// would double the L2 traffic, which at 128 x 256 (3.2 GB for 16384 columns of
// 2030) is the next bound after shared memory -- per stage the MMAs read 147 KB
// of it and the producers write 96 KB, about 1900 cycles against 1660 of the
// tensor pipe.  2030 x 16384 x 2030: 1.87 ms with one 128 x 128 tile whose
// threads staged and issued in turn -> 0.79 ms.  Every wait is bounded; a
// timeout sets an error flag (tc_sgemm_check), writes the tile as NaN and still
// frees the TMEM.
#include <atomic>

#include "common.cuh"
#include "ptx.cuh"

namespace msot {

namespace {

constexpr int GM = 128;          // tile rows (M)
constexpr int GK = 32;           // K per stage
constexpr int G_PROD = 256;      // producer threads
constexpr int G_THREADS = G_PROD + 32;
constexpr int G_APANEL = GM * GK * 4;                                // 16 KB
template <int NT> constexpr int g_bpanel = NT * GK * 4;
template <int NT> constexpr int g_stage = 2 * (G_APANEL + g_bpanel<NT>);
template <int NT> constexpr int g_stages = NT == 256 ? 2 : NT == 128 ? 3 : 4;  // 192 KB each

__device__ int g_gemm_err = 0;

__device__ __forceinline__ uint64_t g_mdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    // start (16 B units) | LBO << 16 | SBO << 32 | descriptor version 1 at
    // bit 46; base offset 0, no swizzle
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor: D F32, A and B TF32, both K-major, N >> 3 at bit
// 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t g_idesc(int M, int N) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// the calling thread's MMAs so far arrive on `bar` when they are done
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
        : "memory");
}
__device__ __forceinline__ float g_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// registers of one stage: A rows m = tid % 128, K groups tid / 128 + 2 j; B in
// units of 8 columns x 4 K groups per warp (a column's 64 bytes are two whole
// sectors, and each 8-lane phase of a 16-byte shared store fills one 128-byte
// core matrix: no bank conflicts)
template <int NT> struct GRegs {
    float4 a[4], b[NT / 32];
};

template <int NT>
__device__ __forceinline__ void g_load(GRegs<NT> &R, const float *A, int lda, const float *B,
                                       int ldb, int M, int N, int K, int m0, int n0, int k0,
                                       bool bvec) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        const int m = m0 + tid % GM;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + 4 * (tid / GM + 2 * j);
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c)
                v[c] = (m < M && k + c < K) ? __ldg(A + (size_t)(k + c) * lda + m) : 0.f;
            R.a[j] = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
#pragma unroll
    for (int j = 0; j < NT / 32; ++j) {
        const int u = j * 8 + warp;
        const int n = n0 + (u >> 1) * 8 + (lane & 7);
        const int k = k0 + 4 * ((u & 1) * 4 + (lane >> 3));
        const float *col = B + (size_t)n * ldb + k;
        if (bvec && k + 3 < K) {
            // past N the last column again: those columns of C are not stored
            R.b[j] = __ldg(reinterpret_cast<const float4 *>(
                B + (size_t)min(n, N - 1) * ldb + min(k, (K - 1) & ~3)));
        } else {
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = (n < N && k + c < K) ? __ldg(col + c) : 0.f;
            R.b[j] = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

__device__ __forceinline__ void g_split_store(const float4 &v, uint8_t *hi, uint8_t *lo,
                                              uint32_t off) {
    const float4 h = make_float4(g_tf32(v.x), g_tf32(v.y), g_tf32(v.z), g_tf32(v.w));
    const float4 l = make_float4(g_tf32(v.x - h.x), g_tf32(v.y - h.y), g_tf32(v.z - h.z),
                                 g_tf32(v.w - h.w));
    *reinterpret_cast<float4 *>(hi + off) = h;
    *reinterpret_cast<float4 *>(lo + off) = l;
}

// element (row r, K group g) of a panel of ROWS rows: core matrix (r / 8, g), row r % 8
template <int ROWS> __device__ __forceinline__ uint32_t g_off(int r, int g) {
    return (uint32_t)(g * (ROWS * 16) + (r >> 3) * 128 + (r & 7) * 16);
}

template <int NT> __device__ __forceinline__ void g_store(const GRegs<NT> &R, uint8_t *stage) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint8_t *ahi = stage, *alo = stage + G_APANEL, *bhi = stage + 2 * G_APANEL,
            *blo = bhi + g_bpanel<NT>;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        g_split_store(R.a[j], ahi, alo, g_off<GM>(tid % GM, tid / GM + 2 * j));
#pragma unroll
    for (int j = 0; j < NT / 32; ++j) {
        const int u = j * 8 + warp;
        g_split_store(R.b[j], bhi, blo,
                      g_off<NT>((u >> 1) * 8 + (lane & 7), (u & 1) * 4 + (lane >> 3)));
    }
}

template <int NT>
__global__ void __launch_bounds__(G_THREADS, 1) k_gemm_3xtf32(
    int M, int N, int K, float alpha, const float *__restrict__ A, int lda,
    const float *__restrict__ B, int ldb, float *__restrict__ C, int ldc, int bvec) {
    constexpr int NS = g_stages<NT>;
    extern __shared__ __align__(1024) uint8_t g_smem[];
    __shared__ __align__(8) uint64_t full[NS], empty[NS], fin;
    __shared__ uint32_t tmem_slot;
    __shared__ int bad;
    const int m0 = blockIdx.x * GM, n0 = blockIdx.y * NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_slot)),
                     "r"((uint32_t)NT));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 32) {
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            mbar_init(smem_u32(&full[i]), G_PROD / 32);
            mbar_init(smem_u32(&empty[i]), 1);
        }
        mbar_init(smem_u32(&fin), 1);
        mbar_init_fence();
        bad = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm = tmem_slot;
    const int ns = (K + GK - 1) / GK;
    if (warp < G_PROD / 32) {
        // producers: the next stage's loads are in flight while this one is
        // split and stored
        auto put = [&](int s, const GRegs<NT> &R) {
            const int buf = s % NS;
            bool ok = true;
            if (s >= NS)  // the MMAs of stage s - NS must be done with this buffer
                ok = mbar_wait_bounded(smem_u32(&empty[buf]), (uint32_t)(s / NS - 1) & 1u);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) bad = 1;
                return false;
            }
            g_store<NT>(R, g_smem + (size_t)buf * g_stage<NT>);
            // generic-proxy stores -> visible to the tensor core (async proxy)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full[buf]));
            return true;
        };
        GRegs<NT> R0, R1;
        g_load<NT>(R0, A, lda, B, ldb, M, N, K, m0, n0, 0, bvec != 0);
        for (int s = 0; s < ns; s += 2) {
            if (s + 1 < ns)
                g_load<NT>(R1, A, lda, B, ldb, M, N, K, m0, n0, (s + 1) * GK, bvec != 0);
            if (!put(s, R0) || s + 1 >= ns) break;
            if (s + 2 < ns)
                g_load<NT>(R0, A, lda, B, ldb, M, N, K, m0, n0, (s + 2) * GK, bvec != 0);
            if (!put(s + 1, R1)) break;
        }
    } else if (lane == 0) {
        int issued = 0;
        for (int s = 0; s < ns; ++s) {
            const int buf = s % NS;
            if (!mbar_wait_bounded(smem_u32(&full[buf]), (uint32_t)(s / NS) & 1u)) {
                bad = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = smem_u32(g_smem + (size_t)buf * g_stage<NT>);
            constexpr uint32_t idesc = g_idesc(GM, NT);
#pragma unroll
            for (int kk = 0; kk < GK / 8; ++kk) {
                const uint32_t ak = (uint32_t)(2 * kk * GM * 16), bk = (uint32_t)(2 * kk * NT * 16);
                const uint32_t bb = base + 2 * G_APANEL + bk;
                const uint64_t ahi = g_mdesc(base + ak, GM * 16, 128);
                const uint64_t alo = g_mdesc(base + G_APANEL + ak, GM * 16, 128);
                const uint64_t bhi = g_mdesc(bb, NT * 16, 128);
                const uint64_t blo = g_mdesc(bb + g_bpanel<NT>, NT * 16, 128);
                const uint64_t da[3] = {ahi, ahi, alo}, db[3] = {bhi, blo, bhi};
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const uint32_t acc = (s | kk | p) != 0;
                    asm volatile(
                        "{\n\t.reg .pred q;\n\t"
                        "setp.ne.b32 q, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, q;\n\t}\n" ::"r"(tm),
                        "l"(da[p]), "l"(db[p]), "r"(idesc), "r"(acc));
                }
            }
            tc_commit(smem_u32(&empty[buf]));
            issued = s + 1;
        }
        // covers every MMA issued before it (and arrives at once if none was)
        tc_commit(smem_u32(&fin));
        if (issued < ns) mbar_wait_bounded(smem_u32(&fin), 0);
    }
    __syncwarp();
    if (!mbar_wait_bounded(smem_u32(&fin), 0)) bad = 1;
    __syncthreads();
    const bool ok = bad == 0;
    if (!ok && threadIdx.x == 0) atomicExch(&g_gemm_err, 1);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // epilogue: producer warp w reads TMEM lanes 32 (w % 4) .. + 31 (rows m) and
    // half of the columns (n); lanes run along m (coalesced stores)
    if (warp < G_PROD / 32) {
        const int m = m0 + (warp & 3) * 32 + lane;
        constexpr int HALF = NT / 2;
#pragma unroll 1
        for (int j0 = (warp >> 2) * HALF; j0 < (warp >> 2) * HALF + HALF; j0 += 16) {
            uint32_t r[16];
            const uint32_t ta = tm + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)j0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, "
                "%10, %11, %12, %13, %14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                  "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                  "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(ta));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (m < M) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int n = n0 + j0 + j;
                    // a tile whose MMAs timed out is written as NaN, never as
                    // a plausible value
                    if (n < N)
                        C[(size_t)n * ldc + m] =
                            ok ? alpha * __uint_as_float(r[j]) : __int_as_float(0x7fc00000);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm),
                     "r"((uint32_t)NT));
}

template <int NT>
static int g_launch(int M, int N, int K, float alpha, const float *A, int lda, const float *B,
                    int ldb, float *C, int ldc, int bvec, cudaStream_t st) {
    constexpr size_t smem = (size_t)g_stages<NT> * g_stage<NT>;
    const cudaError_t e = raise_max_dynamic_smem((const void *)k_gemm_3xtf32<NT>, smem);
    if (e != cudaSuccess) {
        set_error("tc_sgemm: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        return MSOT_ECUDA;
    }
    const dim3 grid((unsigned)div_up(M, GM), (unsigned)div_up(N, NT));
    if (grid.y > 65535u) {
        set_error("tc_sgemm: N = %d too large for one launch", N);
        return MSOT_EINVAL;
    }
    KLAUNCH(k_gemm_3xtf32<NT><<<grid, G_THREADS, smem, st>>>(M, N, K, alpha, A, lda, B, ldb, C,
                                                             ldc, bvec));
    MSOT_LAUNCH_CHECK();
    return MSOT_OK;
}

}  // namespace

int tc_sgemm(int M, int N, int K, float alpha, const float *A, int lda, const float *B, int ldb,
             float *C, int ldc, cudaStream_t st) {
    if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C || lda < M || ldb < K || ldc < M) {
        set_error("tc_sgemm: bad arguments");
        return MSOT_EINVAL;
    }
    // 16-byte B column loads when every column starts 16-byte aligned
    const int bvec = ((reinterpret_cast<uintptr_t>(B) & 15) == 0 && ldb % 4 == 0) ? 1 : 0;
    // the widest tile that still gives every SM one (fewer re-reads and splits
    // of A per column), narrower ones for a few frames
    const long mt = div_up(M, GM), sms = sm_count();
    if (mt * div_up(N, 256) >= sms)
        return g_launch<256>(M, N, K, alpha, A, lda, B, ldb, C, ldc, bvec, st);
    if (mt * div_up(N, 128) >= sms)
        return g_launch<128>(M, N, K, alpha, A, lda, B, ldb, C, ldc, bvec, st);
    return g_launch<64>(M, N, K, alpha, A, lda, B, ldb, C, ldc, bvec, st);
}

int tc_sgemm_check() {
    int v = 0;
    MSOT_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_gemm_err, sizeof v));
    if (v) {
        const int z = 0;
        cudaMemcpyToSymbol(g_gemm_err, &z, sizeof z);
        set_error("tc_sgemm: a bounded wait for the tensor cores ran out");
        return MSOT_ETIMEOUT;
    }
    return MSOT_OK;
}

}  // namespace msot

// Plain matrix product on the CUDA cores: out[M,N] (+)= x[M,K] * W[N,K]^T, float32 accumulate.
//
// This is the 32-bit path of projections of few rows and of sizes that gemm_f32_parts.cu does not take or is not quicker for (no reduced
// precision mode in either), and the plain twin the tensor-core kernels are checked against.
// It also serves mixed operands (bfloat16 activations with a matrix that is stored
// in 32-bit and stays so).  The reference's counterpart is the one-thread-per-row matmul_vec PTX
// kernel (pkg/gpu/cuda/ptx.go:67-129) and ops.MatMulVecInto (pkg/ops/ops.go:30-53).
//
// The order of the additions depends on K alone, so a token's result does not depend on the batch:
// K is cut into four slices of equal length (a multiple of 32, the last may be short or empty), a slice
// is summed with one fused multiply-add after another in ascending k, and the four sums are added as
// (s0 + s1) + (s2 + s3).  Every tile size below keeps this order, so the same bits come from all of them.
//
// A CTA owns a BM x BN tile of the output and has four groups of threads; a group sums one slice of the
// whole tile, with TM x TN outputs per thread, from a ring of STAGES shared-memory stages of
// its own (BK columns of x and W as float32, rows padded by 16 bytes: the float4 reads along k of eight
// neighbouring rows touch all banks once).  Four slices side by side are what keeps a CTA's loads of
// W in flight when M is small and the time is that of reading W; at large M the arithmetic bounds.
// (The tile for many rows, below, has two groups with two slices each.)
#include "common.cuh"

#define SLICES 4

__device__ __forceinline__ int slice_len(int K) { return ((K + SLICES - 1) / SLICES + 31) / 32 * 32; }

__device__ __forceinline__ void gp_cp16(float* smem, const float* gmem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem) : "memory");
}

__device__ __forceinline__ void gp_cp4(float* smem, const float* gmem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a), "l"(gmem) : "memory");
}

template <int THREADS>
__device__ __forceinline__ void group_sync(int g) {
    if (THREADS == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(THREADS) : "memory");
}

// Rows r0.. of a row-major operand into [R][BK + 4] floats; rows from `rows` on and columns from `k_end` on are zero.
// float32 is copied without being waited for: 16 bytes at a time where `chunks` (rows on 16-byte boundaries, K a multiple
// of 4), an element at a time with ELEMENTS.  (A form of the kernel of its own: with both in one, the tiles of up to 64 rows took 10 %
// longer for rows in chunks.)  What is left is loaded, four elements in flight, and converted.
template <typename T, int R, int BK, int THREADS, bool ELEMENTS>
__device__ __forceinline__ void stage_rows(float* dst, const T* src, long long ld, int r0, int rows, int k0, int k_end, int tid,
                                           bool chunks) {
    if (sizeof(T) == 4 && ELEMENTS) {
#pragma unroll 8
        for (int c = tid; c < R * BK; c += THREADS) {
            const int r = c / BK, kk = c % BK;
            float* d = dst + r * (BK + 4) + kk;
            if (r0 + r < rows && k0 + kk < k_end) gp_cp4(d, reinterpret_cast<const float*>(src) + (size_t)(r0 + r) * ld + k0 + kk);
            else *d = 0.f;
        }
    } else if (sizeof(T) == 4 && chunks) {
        constexpr int V = BK / 4;
#pragma unroll
        for (int c = tid; c < R * V; c += THREADS) {
            const int r = c / V, kk = (c % V) * 4;
            float* d = dst + r * (BK + 4) + kk;
            if (r0 + r < rows && k0 + kk < k_end) gp_cp16(d, reinterpret_cast<const float*>(src) + (size_t)(r0 + r) * ld + k0 + kk);
            else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
#pragma unroll 4
        for (int c = tid; c < R * BK; c += THREADS) {
            const int r = c / BK, kk = c % BK;
            float v = 0.f;
            if (r0 + r < rows && k0 + kk < k_end) v = to_f<T>(src[(size_t)(r0 + r) * ld + k0 + kk]);
            dst[r * (BK + 4) + kk] = v;
        }
    }
}

template <typename TX, typename TW, int BM, int BN, int TM, int TN, int BK, int STAGES, bool ELEMENTS>
__global__ void __launch_bounds__((BM / TM) * (BN / TN) * SLICES) gemm_plain_kernel(
    const TX* x, const TW* __restrict__ w, void* out, int out_bf16, int accumulate, int M, int N, int K, long long ldx,
    long long ldo, const float* __restrict__ bias, int m_tiles, int async_x, int async_w, int early) {
    constexpr int THN = BN / TN, THM = BM / TM, THREADS = THN * THM;
    constexpr int STAGE = (BM + BN) * (BK + 4);
    extern __shared__ __align__(16) float sm[];
    if (early) pdl_launch();
    const int g = threadIdx.x / THREADS, tid = threadIdx.x % THREADS;
    const int tx = tid % THN, ty = tid / THN;
    const int m0 = (int)(blockIdx.x % m_tiles) * BM, n0 = (int)(blockIdx.x / m_tiles) * BN;
    const int len = slice_len(K);
    const int k_begin = min(K, g * len), k_end = min(K, (g + 1) * len);
    const int steps = (k_end - k_begin + BK - 1) / BK;
    float* ring = sm + (size_t)g * STAGES * STAGE;
    auto load_w = [&](int it) {
        if (it < steps) stage_rows<TW, BN, BK, THREADS, ELEMENTS>(ring + (it % STAGES) * STAGE + BM * (BK + 4), w, K, n0, N, k_begin + it * BK, k_end, tid, async_w);
    };
    auto load_x = [&](int it) {
        if (it < steps) stage_rows<TX, BM, BK, THREADS, ELEMENTS>(ring + (it % STAGES) * STAGE, x, ldx, m0, M, k_begin + it * BK, k_end, tid, async_x);
    };
#pragma unroll 1
    for (int s = 0; s < STAGES - 1; ++s) load_w(s);     // weights: nothing before this kernel writes them
    pdl_wait();
#pragma unroll 1
    for (int s = 0; s < STAGES - 1; ++s) {
        load_x(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll 1
    for (int it = 0; it < steps; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        group_sync<THREADS>(g);                          // stage `it` is there, and nobody reads stage it - 1 any more
        load_w(it + STAGES - 1);
        load_x(it + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* xs = ring + (it % STAGES) * STAGE + ty * (BK + 4);
        const float* ws = ring + (it % STAGES) * STAGE + (BM + tx) * (BK + 4);
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float4 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * THN * (BK + 4) + kk);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(xs + i * THM * (BK + 4) + kk);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
            }
        }
    }
    // the groups' sums through shared memory: (s0 + s1) + (s2 + s3)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (g > 0) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) sm[((g - 1) * TM * TN + i * TN + j) * THREADS + tid] = acc[i][j];
    }
    __syncthreads();
    if (g > 0) return;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + i * THM;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * THN;
            if (m >= M || n >= N) continue;
            const float* o = sm + (i * TN + j) * THREADS + tid;
            float v = acc[i][j] + o[0];
            v += o[TM * TN * THREADS] + o[2 * TM * TN * THREADS];
            if (bias != nullptr) v += bias[n];
            if (out_bf16) reinterpret_cast<bf16*>(out)[(size_t)m * ldo + n] = __float2bfloat16_rn(v);
            else {
                float* p = reinterpret_cast<float*>(out) + (size_t)m * ldo + n;
                *p = accumulate ? *p + v : v;
            }
        }
    }
}

template <typename TX, typename TW, int BM, int BN, int TM, int TN, int BK, int STAGES, bool ELEMENTS = false>
static int launch_tile(const TX* x, const TW* w, void* out, int out_bf16, int accumulate, int M, int N, int K,
                       long long ldx, long long ldo, const float* bias, cudaStream_t stream) {
    constexpr int threads = (BM / TM) * (BN / TN) * SLICES;
    constexpr size_t ring = (size_t)SLICES * STAGES * (BM + BN) * (BK + 4) * sizeof(float);
    static_assert(ring <= 227 * 1024 && ring >= (size_t)(SLICES - 1) * BM * BN * sizeof(float), "shared memory");
    auto kern = gemm_plain_kernel<TX, TW, BM, BN, TM, TN, BK, STAGES, ELEMENTS>;
    static int known[GG_MAX_DEVICES] = {};
    int resident = 0;
    const int rc = gg_resident(kern, threads, ring, known, resident);
    if (rc != 0) return rc;
    const int m_tiles = (M + BM - 1) / BM;
    const long long tiles = (long long)m_tiles * ((N + BN - 1) / BN);
    if (tiles > 0x7fffffffLL) return GG_ERR_ARG;
    const int async_x = sizeof(TX) == 4 && K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)x & 15) == 0;
    const int async_w = sizeof(TW) == 4 && K % 4 == 0 && ((uintptr_t)w & 15) == 0;
    // the successor may start early only where no CTA of this grid still waits for an SM (see common.cuh)
    return gg_launch(kern, dim3((unsigned)tiles), dim3(threads), ring, stream, 1, x, w, out, out_bf16, accumulate, M, N, K, ldx, ldo,
                     bias, m_tiles, async_x, async_w, (int)(tiles <= resident));
}

// ----------------------------------------------------------------------------- the tile for many rows
// BM x 64 outputs, two groups of BM threads with two slices each, 8 x 8 outputs a thread.  Here the multipliers bound, and
// on sm_100a they reach their rate only with the packed form (measured, registers only: fma.rn.f32 60 TFLOP/s,
// fma.rn.f32x2 74): a thread's sums are pairs of neighbouring columns.  So x and W lie in shared memory with k as the
// slow index, four columns or rows a 16-byte read, and come there through registers (the next stage's loads are
// issued before this stage's arithmetic).  Shared-memory reads bound it next: with x stored as pairs, which saves packing each
// value twice but reads six times 16 bytes a column instead of four, a prompt batch took 6.29 ms instead of 4.97.  Both halves of a
// packed multiply-add are rounded as fma.rn.f32, so the bits are those of the other tiles.
#define WIDE_BN 64
#define WIDE_BK 16

// This thread's part of a stage, R rows of WIDE_BK columns, into registers as it lies in memory (a conversion would wait for the load):
// VEC (rows of four elements aligned): columns 4 (tid % 4) .. + 3 of rows tid / 4 + THREADS / 4 i; else column tid % 16 of rows
// tid / 16 + THREADS / 16 j, so that a warp's loads are two runs of neighbours.
template <typename T, int R, int THREADS, bool VEC>
__device__ __forceinline__ void wide_load(T (&v)[R * WIDE_BK / THREADS], const T* src, long long ld, int r0, int rows, int k0, int k_end,
                                          int tid) {
    constexpr int PER = R * WIDE_BK / THREADS;
    if (VEC) {
        const int k = k0 + tid % 4 * 4;
#pragma unroll
        for (int i = 0; i < PER / 4; ++i) {
            const int r = r0 + tid / 4 + THREADS / 4 * i;
            const bool in = r < rows && k < k_end;
            const T* p = src + (size_t)r * ld + k;
            if (sizeof(T) == 4) *reinterpret_cast<uint4*>(&v[4 * i]) = in ? *reinterpret_cast<const uint4*>(p) : make_uint4(0u, 0u, 0u, 0u);
            else *reinterpret_cast<uint2*>(&v[4 * i]) = in ? *reinterpret_cast<const uint2*>(p) : make_uint2(0u, 0u);
        }
    } else {
        const int k = k0 + tid % 16;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int r = r0 + tid / 16 + THREADS / 16 * j;
            v[j] = r < rows && k < k_end ? src[(size_t)r * ld + k] : from_f<T>(0.f);
        }
    }
}
// and from there to shared memory as float32, k as the slow index, rows of LD floats
template <typename T, int R, int THREADS, int LD, bool VEC>
__device__ __forceinline__ void wide_store(float* dst, const T (&v)[R * WIDE_BK / THREADS], int tid) {
    constexpr int PER = R * WIDE_BK / THREADS;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (VEC) dst[(tid % 4 * 4 + j % 4) * LD + tid / 4 + THREADS / 4 * (j / 4)] = to_f<T>(v[j]);
        else dst[tid % 16 * LD + tid / 16 + THREADS / 16 * j] = to_f<T>(v[j]);
    }
}
__device__ __forceinline__ unsigned long long gp_pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 gp_unpack(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

template <typename TX, typename TW, int BM, bool VEC>
__global__ void __launch_bounds__(2 * BM) gemm_plain_wide_kernel(
    const TX* x, const TW* __restrict__ w, void* out, int out_bf16, int accumulate, int M, int N, int K, long long ldx,
    long long ldo, const float* __restrict__ bias, int m_tiles, int early) {
    constexpr int BN = WIDE_BN, BK = WIDE_BK, LX = BM + 4, LW = BN + 4, STAGE = BK * (LX + LW);
    extern __shared__ __align__(16) float sm[];
    if (early) pdl_launch();
    const int g = threadIdx.x / BM, tid = threadIdx.x % BM;
    const int tx = tid % 8, ty = tid / 8;               // columns 4 tx + {0..3, 32..35}, rows 4 ty + {0..3, BM/2..}
    const int m0 = (int)(blockIdx.x % m_tiles) * BM, n0 = (int)(blockIdx.x / m_tiles) * BN;
    const int len = slice_len(K);
    const int k_begin = min(K, g * 2 * len), k_end = min(K, (g + 1) * 2 * len);
    const int steps = (k_end - k_begin + BK - 1) / BK, per_slice = len / BK;
    float* ring = sm + (size_t)g * 2 * STAGE;
    alignas(16) TX xr[BK];
    alignas(16) TW wr[BN * BK / BM];
    auto load_w = [&](int it) { wide_load<TW, BN, BM, VEC>(wr, w, K, n0, N, k_begin + it * BK, k_end, tid); };
    auto load_x = [&](int it) { wide_load<TX, BM, BM, VEC>(xr, x, ldx, m0, M, k_begin + it * BK, k_end, tid); };
    auto store = [&](int it) {
        float* xs = ring + (it & 1) * STAGE;
        wide_store<TX, BM, BM, LX, VEC>(xs, xr, tid);
        wide_store<TW, BN, BM, LW, VEC>(xs + BK * LX, wr, tid);
    };
    unsigned long long acc[8][4], run[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    if (steps > 0) load_w(0);
    pdl_wait();
    if (steps > 0) { load_x(0); store(0); }
    group_sync<BM>(g);
#pragma unroll 1
    for (int it = 0; it < steps; ++it) {
        if (it + 1 < steps) { load_w(it + 1); load_x(it + 1); }
        if (it == per_slice) {                           // the first of the group's two slices is done
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { run[i][j] = acc[i][j]; acc[i][j] = 0ull; }
        }
        const float* xs = ring + (it & 1) * STAGE + 4 * ty;
        const float* ws = ring + (it & 1) * STAGE + BK * LX + 4 * tx;
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(ws + k * LW), b1 = *reinterpret_cast<const ulonglong2*>(ws + k * LW + 32);
            const unsigned long long b[4] = {b0.x, b0.y, b1.x, b1.y};
            const float4 a0 = *reinterpret_cast<const float4*>(xs + k * LX), a1 = *reinterpret_cast<const float4*>(xs + k * LX + BM / 2);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long aa = gp_pack(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(b[j]));
            }
        }
        if (it + 1 < steps) store(it + 1);               // (its last readers left it a barrier ago)
        group_sync<BM>(g);
    }
    float f[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float2 v = gp_unpack(acc[i][j]);
            if (steps > per_slice) {
                const float2 r = gp_unpack(run[i][j]);
                v.x = r.x + v.x; v.y = r.y + v.y;
            }
            f[i][2 * j] = v.x; f[i][2 * j + 1] = v.y;
        }
    __syncthreads();
    if (g > 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) sm[(i * 8 + j) * BM + tid] = f[i][j];
    }
    __syncthreads();
    if (g > 0) return;
    const bool vec_o = !out_bf16 && (ldo & 3) == 0 && (((uintptr_t)out) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + 4 * ty + (i & 3) + (i >> 2) * (BM / 2);
        if (m >= M) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = n0 + 4 * tx + 32 * h;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[j] = f[i][4 * h + j] + sm[(i * 8 + 4 * h + j) * BM + tid];
                if (bias != nullptr && n + j < N) v[j] += bias[n + j];
            }
            if (vec_o && n + 4 <= N) {
                float4* p = reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + (size_t)m * ldo + n);
                float4 r = make_float4(v[0], v[1], v[2], v[3]);
                if (accumulate) { const float4 o = *p; r.x += o.x; r.y += o.y; r.z += o.z; r.w += o.w; }
                *p = r;
                continue;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n + j >= N) continue;
                if (out_bf16) reinterpret_cast<bf16*>(out)[(size_t)m * ldo + n + j] = __float2bfloat16_rn(v[j]);
                else {
                    float* p = reinterpret_cast<float*>(out) + (size_t)m * ldo + n + j;
                    *p = accumulate ? *p + v[j] : v[j];
                }
            }
        }
    }
}

template <typename TX, typename TW, int BM, bool VEC>
static int launch_wide_as(const TX* x, const TW* w, void* out, int out_bf16, int accumulate, int M, int N, int K,
                       long long ldx, long long ldo, const float* bias, cudaStream_t stream) {
    constexpr size_t ring = (size_t)4 * WIDE_BK * (BM + WIDE_BN + 8) * sizeof(float);
    static_assert(ring >= (size_t)64 * BM * sizeof(float), "the second group's sums go through the stages");
    auto kern = gemm_plain_wide_kernel<TX, TW, BM, VEC>;
    static int known[GG_MAX_DEVICES] = {};
    int resident = 0;
    const int rc = gg_resident(kern, 2 * BM, ring, known, resident);
    if (rc != 0) return rc;
    const int m_tiles = (M + BM - 1) / BM;
    const long long tiles = (long long)m_tiles * ((N + WIDE_BN - 1) / WIDE_BN);
    if (tiles > 0x7fffffffLL) return GG_ERR_ARG;
    return gg_launch(kern, dim3((unsigned)tiles), dim3(2 * BM), ring, stream, 1, x, w, out, out_bf16, accumulate, M, N, K, ldx, ldo,
                     bias, m_tiles, (int)(tiles <= resident));
}

template <typename TX, typename TW, int BM>
static int launch_wide(const TX* x, const TW* w, void* out, int out_bf16, int accumulate, int M, int N, int K,
                       long long ldx, long long ldo, const float* bias, cudaStream_t stream) {
    const bool vec = K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)x & (sizeof(TX) * 4 - 1)) == 0 && ((uintptr_t)w & (sizeof(TW) * 4 - 1)) == 0;
    if (vec) return launch_wide_as<TX, TW, BM, true>(x, w, out, out_bf16, accumulate, M, N, K, ldx, ldo, bias, stream);
    return launch_wide_as<TX, TW, BM, false>(x, w, out, out_bf16, accumulate, M, N, K, ldx, ldo, bias, stream);
}

template <typename TX, typename TW>
static int launch(const void* xv, const void* wv, void* out, int out_bf16, int accumulate,
                  int M, int N, int K, long long ldx, long long ldo, const float* bias, cudaStream_t stream) {
    const TX* x = (const TX*)xv;
    const TW* w = (const TW*)wv;
#define GP(BM, BN, TM, TN, BK, ...) return launch_tile<TX, TW, BM, BN, TM, TN, BK, __VA_ARGS__>(x, w, out, out_bf16, accumulate, M, N, K, ldx, ldo, bias, stream)
    // Up to 16 rows the time is that of reading W, and what counts is how much of it is asked for at a time.  With a CTA an SM
    // or less, deep rings of wide stages; with more tiles, the ring that lets most of them be resident.  Measured, M = 4
    // (us; BK 32 in 6 stages for all | as below): 2,048 x 2,048 10.7 | 6.4, 2,048 x 5,376 25.4 | 13.6, 4,096 x 2,048 11.6 | 9.3,
    // 10,752 x 2,048 25.2 | 22.2, 65,536 x 2,048 106 | 98 (5.5 TB/s).
    const long long tiles = (long long)((N + 15) / 16) * ((M + 15) / 16);
    if (M <= 2) {
        if (tiles <= 148) GP(2, 16, 1, 1, 128, 4);
        if (tiles <= 296) GP(2, 16, 1, 1, 64, 4);
        GP(2, 16, 1, 1, 64, 2);
    }
    if (M <= 4) {
        if (tiles <= 148) GP(4, 16, 2, 1, 128, 4);
        if (tiles <= 296) GP(4, 16, 2, 1, 64, 4);
        GP(4, 16, 2, 1, 64, 2);
    }
    if (M <= 8) {
        if (tiles <= 74) GP(8, 8, 2, 1, 128, 3);
        if (tiles <= 148) GP(8, 16, 2, 2, 64, 6);
        if (tiles <= 296) GP(8, 16, 2, 2, 64, 4);
        GP(8, 16, 2, 2, 64, 2);
    }
    if (M <= 16) {
        if (tiles <= 148) GP(16, 8, 2, 2, 64, 3);
        if (tiles <= 296) GP(16, 16, 4, 2, 64, 3);
        GP(16, 16, 4, 2, 64, 2);
    }
    // More rows: the quickest of four tiles.  Measured per tile, in microseconds per 1,000 of K: 148 tiles or fewer, and 296 (two an
    // SM); a grid is as many rounds of 296 and one of what is left.  Three rows of the table: float32 in chunks, float32 by elements, any
    // bfloat16 operand.  Over 352 products (17 to 2,048 rows, ten matrices) the choice is within 1 % of the best tile on average
    // and 25 % at worst; one share of the multipliers' rate per tile, whatever the operands, was 12 % and 211 %.
    static const float round_us[3][4][2] = {{{11, 11}, {30, 35}, {42, 55}, {54, 110}},
                                            {{12, 21}, {27, 59}, {62, 70}, {60, 120}},
                                            {{16, 23}, {38, 48}, {57, 76}, {60, 130}}};
    const bool elements = (sizeof(TX) == 4 && (K % 4 || ldx % 4 || ((uintptr_t)x & 15))) || (sizeof(TW) == 4 && (K % 4 || ((uintptr_t)w & 15)));
    const float (*us)[2] = round_us[sizeof(TX) == 2 || sizeof(TW) == 2 ? 2 : (int)elements];
    const int rows[4] = {32, 64, 64, 128}, cols[4] = {16, 32, 64, 64};
    int best = 0;
    float least = 0.f;
    for (int i = 0; i < 4; ++i) {
        const long long t = (long long)((M + rows[i] - 1) / rows[i]) * ((N + cols[i] - 1) / cols[i]), left = t % 296;
        const float cost = us[i][1] * (float)(t / 296) + (left == 0 ? 0.f : us[i][left > 148]);
        if (i == 0 || cost < least) { best = i; least = cost; }
    }
    if (best == 0) {
        if (elements) GP(32, 16, 4, 4, 32, 4, true);
        GP(32, 16, 4, 4, 32, 4, false);
    }
    if (best == 1) {
        if (elements) GP(64, 32, 8, 4, 16, 3, true);
        GP(64, 32, 8, 4, 16, 3, false);
    }
    if (best == 2) return launch_wide<TX, TW, 64>(x, w, out, out_bf16, accumulate, M, N, K, ldx, ldo, bias, stream);
    return launch_wide<TX, TW, 128>(x, w, out, out_bf16, accumulate, M, N, K, ldx, ldo, bias, stream);
#undef GP
}

// x[M, K] with row stride ldx (elements), w[N, K] contiguous, out[M, N] with row stride ldo.
// accumulate != 0: out += product (float32 out only; this is the residual add).  bias (may be null): [N] float32.
GG_API gg_gemm_plain(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                     int accumulate, int M, int N, int K, long long ldx, long long ldo, const float* bias,
                     cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || ldx < K || ldo < N) return GG_ERR_ARG;
    if ((M + 63) / 64 > 65535) return GG_ERR_ARG;
    if (out_dtype != GG_F32 && out_dtype != GG_BF16) return GG_ERR_DTYPE;
    if (out_dtype == GG_BF16 && accumulate) return GG_ERR_DTYPE;  // sums are kept in float32
    const int ob = out_dtype == GG_BF16;
    if (x_dtype == GG_F32 && w_dtype == GG_F32) return launch<float, float>(x, w, out, ob, accumulate, M, N, K, ldx, ldo, bias, stream);
    if (x_dtype == GG_BF16 && w_dtype == GG_BF16) return launch<bf16, bf16>(x, w, out, ob, accumulate, M, N, K, ldx, ldo, bias, stream);
    if (x_dtype == GG_BF16 && w_dtype == GG_F32) return launch<bf16, float>(x, w, out, ob, accumulate, M, N, K, ldx, ldo, bias, stream);
    if (x_dtype == GG_F32 && w_dtype == GG_BF16) return launch<float, bf16>(x, w, out, ob, accumulate, M, N, K, ldx, ldo, bias, stream);
    return GG_ERR_DTYPE;
}

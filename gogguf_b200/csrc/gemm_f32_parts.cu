// 32-bit matrix product of many rows on the tensor cores: out[M,N] (+)= x[M,K] * W[N,K]^T (+ bias), all float32.
//
// A float32 number is the sum of three bfloat16 numbers without a rest: the nearest one, the one nearest to what that leaves, and
// what is left then (its 24 bits are 8, 8 and 8 with a sign each).  So a product of two is nine products of parts, of which the six down
// to 2^-16 of the first are taken.  The second part is at most 2^-8 of a number and the third at most 2^-17, so the three left out
// are below 2^-24 of the product together, the rounding of a 32-bit product, and have no sign of their own (4 million products of
// normal numbers: 0.87 x 2^-24 at most, 0.10 in the mean square, where a rounding has 0.42).  Each product taken is exact in the
// tensor core's multiplier.  (Parts by rounding, and sums kept outside the tensor core: Henry, Tang and Heinecke 2019, Ootomo and
// Yokota 2022.)  What the tensor core does not do is round: it cuts off what an addition shifts out, and over a long contraction
// that drift would be larger than the rounding of the CUDA cores' sums (2.1e-6 against 0.8e-6 at K = 2,048).  So the accumulator
// in tensor memory holds 32 columns of K at a time, the small products first and the two large ones (16 columns an instruction)
// last, and every 32 columns' sum is added in registers, rounded to nearest.
// Relative error against 64 bits, gemm_plain.cu | here (1e-7), K = 256, 2,048, 5,376: normal operands 1.5 | 0.75, 4.0 | 1.0, 6.5 | 1.1; of one
// sign 0.72 | 0.67, 1.8 | 0.84, 2.6 | 0.78; one channel a hundred times the others 1.7 | 0.70, 4.6 | 1.2, 7.2 | 1.2.  A row with one term alone
// is what the CUDA cores round once and the tensor core cuts off: 0.25 | 0.45, at most 2.3 x 2^-24 of the term.
//
// Bounds: six products at the dense bfloat16 rate are 280 TFLOP/s of 32-bit products, where packed multiply-adds on the CUDA cores
// have 74 (and reach 41, bound by reads of shared memory).  Measured, 450 rows (us, gemm_plain.cu | this): 4,096 x 2,048 226 | 51,
// 10,752 x 2,048 547 | 113, 2,048 x 5,376 287 | 59; 17 rows: 23 | 19, 68 | 40, 52 | 24.
//
// A CTA owns 128 rows of W (the instruction's M) and BN rows of x, over the whole of K or a share of it, and has
//   warp 0      TMA: W as float32 (two boxes of 128 x 32 a stage), the three parts of x (BN x 64 each; split_rows_kernel makes them);
//   warp 1      the products: parts of W from tensor memory, parts of x from shared memory;
//   warps 2-5   W's parts: a row a thread, 32 columns at a time from shared memory to tensor memory.  W is split here, once for every
//               tile of x, because its parts would be half as much again to keep and to read;
//   warps 6-13  the sums: BN / 2 of a row's outputs a thread.
// Grids of at most one CTA an SM walk over (tile, share) items.  Where shares of K are summed by several CTAs, their sums lie in scratch
// and finish_kernel adds them in the order of K.
//
// Infinities and NaN: parts of an infinity are an infinity and NaN, and a zero part times an infinity is NaN, so a product of parts is
// not finite wherever the 32-bit product is not; nor is it where an operand is so large that its first part rounds to an
// infinity.  Every sum that is not finite is made again from the operands, by multiply-adds, and is what those give (plain_sums).  Parts
// below 2^-133 are cut off, an absolute error of that size per operand.
//
// Rows of x are taken in slabs, so that their parts fill 256 MB of scratch at most.
#include <initializer_list>
#include "common.cuh"
#include "tma_util.cuh"

namespace {

constexpr int ROWS = 128;                 // of W in a tile
constexpr int STEP = 64;                  // columns of K in a stage
constexpr int CHUNK = 32;                 // columns of K that are summed in tensor memory
constexpr int W_BYTES = ROWS * STEP * 4;
constexpr int THREADS = 448;
constexpr int PART_COLS = CHUNK / 2;      // 32-bit columns of tensor memory that hold a part of 32 columns of K
constexpr int A_COLS = 3 * PART_COLS;

struct Shape {
    int M, N, K;
    int m_tiles, n_tiles, shares, steps;  // steps: stages in a share of K (the last share may have fewer)
    int items;
};

// The sums of four rows of x with four rows of w by multiply-adds, a warp's lanes along k; a lane gets the four of w's row lane % 4.
// (450 rows with an infinity each by 10,752 x 2,048: 3.1 ms; 44.7 with a thread's walk over K for each of its sums, 0.55 in gemm_plain.cu.
// With a NaN each: 0.29, rows_with_nan.)
__device__ __forceinline__ float4 plain_sums(const float* x, long long ldx, int x_rows, int vec, const float* w, int ldw, int w_rows, int k0, int k1) {
    const int lane = threadIdx.x & 31;
    const float* xr[4];
    const float* wr[4];
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        xr[i] = x + (size_t)min(i, x_rows - 1) * ldx;
        wr[i] = w + (size_t)min(i, w_rows - 1) * ldw;
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
    }
#pragma unroll 2
    for (int k = k0 + 4 * lane; k < k1; k += 128) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            b[i] = *reinterpret_cast<const float4*>(wr[i] + k);
            if (vec) a[i] = *reinterpret_cast<const float4*>(xr[i] + k);
            else a[i] = make_float4(xr[i][k], xr[i][k + 1], xr[i][k + 2], xr[i][k + 3]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                s[i][j] = fmaf(a[j].w, b[i].w, fmaf(a[j].z, b[i].z, fmaf(a[j].y, b[i].y, fmaf(a[j].x, b[i].x, s[i][j]))));
    }
    float4 mine = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 t = make_float4(warp_sum(s[i][0]), warp_sum(s[i][1]), warp_sum(s[i][2]), warp_sum(s[i][3]));
        if ((lane & 3) == i) mine = t;
    }
    return mine;
}

// Which of four rows of x have a NaN among their columns k0 .. k1: their sums are NaN whatever w holds.
__device__ __forceinline__ uint32_t rows_with_nan(const float* x, long long ldx, int x_rows, int vec, int k0, int k1) {
    uint32_t found = 0u;
#pragma unroll 4
    for (int k = k0 + 4 * (int)(threadIdx.x & 31); k < k1; k += 128)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* r = x + (size_t)min(i, x_rows - 1) * ldx + k;
            float4 v;
            if (vec) v = *reinterpret_cast<const float4*>(r);
            else v = make_float4(r[0], r[1], r[2], r[3]);
            if (v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w) found |= 1u << i;
        }
    return __reduce_or_sync(0xffffffffu, found);
}

// Where a warp's sums of 32 columns (outputs of rows m .. of x with rows n .. + 31 of w) are made again.
struct Again {
    const float* x;
    const float* w;
    float* out;               // [row of x][row of w]
    long long ldx, ldo;
    int M, N, K, k0, k1, accumulate;
    float bias;               // the lane's
};
// The warp's outputs whose bits are set in its lanes' words.  (Not inlined, and its numbers by reference: the registers would be the kernel's.)
__device__ __noinline__ void make_again(uint32_t bits, int m, int n, const Again& a) {
    const int lane = threadIdx.x & 31, vec = a.ldx % 4 == 0 && ((uintptr_t)a.x & 15) == 0;
    for (int j = 0; j < 32; j += 4) {
        uint32_t mine = bits >> j & 15u;
        if (!__any_sync(0xffffffffu, mine != 0u)) continue;
        const uint32_t nan = rows_with_nan(a.x + (size_t)(m + j) * a.ldx, a.ldx, a.M - m - j, vec, a.k0, a.k1);
        for (uint32_t left = mine & nan; left != 0u; left &= left - 1u)
            a.out[(size_t)(m + j + __ffs(left) - 1) * a.ldo + n + lane] = __int_as_float(0x7fffffff);
        mine &= ~nan;
        uint32_t rows = __ballot_sync(0xffffffffu, mine != 0u);
        while (rows != 0u) {                                         // four neighbouring rows of w at a time
            const int r = (__ffs(rows) - 1) & ~3;
            rows &= ~(15u << r);
            __syncwarp();
            const float4 t = plain_sums(a.x + (size_t)(m + j) * a.ldx, a.ldx, a.M - m - j, vec, a.w + (size_t)(n + r) * a.K, a.K, a.N - n - r, a.k0, a.k1);
            if ((lane & ~3) != r) continue;
            const float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!(mine >> u & 1u)) continue;
                float* p = a.out + (size_t)(m + j + u) * a.ldo + n + lane;
                *p = a.accumulate ? *p + (v[u] + a.bias) : v[u] + a.bias;
            }
        }
    }
}

// a, b -> their three parts, two neighbours along k in a word.  The third part is what is left: its 8 bits stand in the upper half of a
// float32 already.
__device__ __forceinline__ uint32_t nearest_pair(float a, float b) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&t);
}
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    p0 = nearest_pair(a, b);
    a -= __uint_as_float(p0 << 16);
    b -= __uint_as_float(p0 & 0xffff0000u);
    p1 = nearest_pair(a, b);
    a -= __uint_as_float(p1 << 16);
    b -= __uint_as_float(p1 & 0xffff0000u);
    p2 = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// parts[p][m][k], rows of ld elements (K rounded up to 8; what lies between is not read).  Four columns a thread.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* x, long long ldx, bf16* __restrict__ parts, int M, int K, int ld, int vec) {
    pdl_launch();
    pdl_wait();
    const int per_row = K / 4;
    const long long total = (long long)M * per_row, plane = (long long)M * ld;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const int m = (int)(i / per_row), k = (int)(i % per_row) * 4;
        const float* src = x + (size_t)m * ldx + k;
        float4 v;
        if (vec) v = *reinterpret_cast<const float4*>(src);
        else v = make_float4(src[0], src[1], src[2], src[3]);
        uint32_t a[3], b[3];
        split_pair(v.x, v.y, a[0], a[1], a[2]);
        split_pair(v.z, v.w, b[0], b[1], b[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(parts + p * plane + (size_t)m * ld + k) = make_uint2(a[p], b[p]);
    }
}

template <int BN, int STAGES, int PARTS>
__global__ void __launch_bounds__(THREADS, 1) parts_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                           const float* x, long long ldx, const float* __restrict__ w, float* out, long long ldo,
                                                           int accumulate, const float* __restrict__ bias, float* partial, const Shape sh,
                                                           int* __restrict__ status) {
    constexpr int X_PART = BN * STEP * 2, STAGE_BYTES = W_BYTES + 3 * X_PART, HALF = BN / 2;
    static_assert(BN % 32 == 0 && 2 * BN + PARTS * A_COLS <= 512, "tensor memory");
    extern __shared__ uint8_t raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_w = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t* full_x = full_w + STAGES;
    uint64_t* empty = full_x + STAGES;          // the converting threads and the products' commit
    uint64_t* a_full = empty + STAGES;          // [PARTS]
    uint64_t* a_empty = a_full + PARTS;
    uint64_t* acc_full = a_empty + PARTS;       // [2]
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    pdl_launch();        // the grid is resident as a whole
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { tma::mbar_init(&full_w[s], 1); tma::mbar_init(&full_x[s], 1); tma::mbar_init(&empty[s], 129); }
        for (int b = 0; b < PARTS; ++b) { tma::mbar_init(&a_full[b], 128); tma::mbar_init(&a_empty[b], 1); }
        for (int b = 0; b < 2; ++b) { tma::mbar_init(&acc_full[b], 1); tma::mbar_init(&acc_empty[b], 256); }
        *abort_flag = 0;
        tma::mbar_fence_init();
        tma::prefetch_map(&map_w);
        tma::prefetch_map(&map_x);
    }
    if (warp == 1) tc5::alloc(tmem_slot, 512);
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    const uint32_t tmem = *tmem_slot;
    const int all_steps = (sh.K + STEP - 1) / STEP;
    auto place = [&](int item, int& m0, int& n0, int& step0, int& n_steps, int& share) {
        m0 = item % sh.m_tiles * BN;
        const int r = item / sh.m_tiles;
        share = r % sh.shares;
        n0 = r / sh.shares * ROWS;
        step0 = share * sh.steps;
        n_steps = min(sh.steps, all_steps - step0);
    };
    int m0, n0, step0, n_steps, share;

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            auto load_w = [&](int s, int step) {
                tma::mbar_expect_tx(&full_w[s], W_BYTES);
                tma::load_2d(smem + s * STAGE_BYTES, &map_w, &full_w[s], step * STEP, n0);
                tma::load_2d(smem + s * STAGE_BYTES + W_BYTES / 2, &map_w, &full_w[s], step * STEP + 32, n0);
            };
            auto load_x = [&](int s, int step) {
                tma::mbar_expect_tx(&full_x[s], 3 * X_PART);
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    tma::load_2d(smem + s * STAGE_BYTES + W_BYTES + p * X_PART, &map_x, &full_x[s], step * STEP, p * sh.M + m0);
            };
            for (int item = blockIdx.x; item < sh.items && ok; item += gridDim.x) {
                place(item, m0, n0, step0, n_steps, share);
                int i = 0;
                if (it == 0) {                  // weights ahead of the wait: no kernel writes them
                    const int pre = min(n_steps, STAGES);
                    for (; i < pre; ++i) load_w(i, step0 + i);
                    pdl_wait();
                    for (int j = 0; j < pre; ++j) load_x(j, step0 + j);
                    it = pre;
                }
                for (; i < n_steps; ++i, ++it) {
                    const int s = it % STAGES;
                    if (!tma::mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, abort_flag, status, 1)) { ok = false; break; }
                    load_w(s, step0 + i);
                    load_x(s, step0 + i);
                }
            }
            if (it == 0) pdl_wait();
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = tc5::idesc_bf16(ROWS, BN, 0);
            int it = 0, c = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < sh.items && ok; item += gridDim.x) {
                place(item, m0, n0, step0, n_steps, share);
                for (int i = 0; i < n_steps && ok; ++i, ++it) {
                    const int s = it % STAGES;
                    ok = tma::mbar_wait(&full_x[s], (it / STAGES) & 1, abort_flag, status, 2);
                    for (int h = 0; h < 2 && ok; ++h, ++c) {
                        const int pb = c % PARTS, ab = c & 1;
                        ok = tma::mbar_wait(&a_full[pb], (c / PARTS) & 1, abort_flag, status, 2)
                             && tma::mbar_wait(&acc_empty[ab], ((c >> 1) & 1) ^ 1, abort_flag, status, 4);
                        if (!ok) break;
                        tc5::fence_after();
                        const uint32_t acc = tmem + (uint32_t)(ab * BN), a = tmem + (uint32_t)(2 * BN + pb * A_COLS);
                        const uint32_t xs = tma::smem_u32(smem + s * STAGE_BYTES + W_BYTES) + (uint32_t)(h * 64);
                        // the small products first: what the tensor core cuts off is a part of the larger addend
                        constexpr int PW[6] = {0, 1, 2, 0, 1, 0}, PX[6] = {2, 1, 0, 1, 0, 0};
#pragma unroll
                        for (int q = 0; q < 6; ++q)
#pragma unroll
                            for (int k = 0; k < 2; ++k)
                                tc5::mma_a_tmem(acc, a + (uint32_t)(PW[q] * PART_COLS + 8 * k),
                                                tc5::smem_desc(xs + (uint32_t)(PX[q] * X_PART + 32 * k), 16, 1024), idesc, q + k > 0 ? 1u : 0u);
                        tc5::commit(&a_empty[pb]);
                        tc5::commit(&acc_full[ab]);
                    }
                    if (ok) tc5::commit(&empty[s]);
                }
            }
        }
    } else if (warp < 6) {
        const int row = (warp & 3) * 32 + lane;
        int it = 0, c = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < sh.items && ok; item += gridDim.x) {
            place(item, m0, n0, step0, n_steps, share);
            for (int i = 0; i < n_steps && ok; ++i, ++it) {
                const int s = it % STAGES;
                // (a warp's waits may end apart when one runs out; what follows is the whole warp's)
                ok = __all_sync(0xffffffffu, tma::mbar_wait(&full_w[s], (it / STAGES) & 1, abort_flag, status, 3));
                for (int h = 0; h < 2 && ok; ++h, ++c) {
                    const uint8_t* src = smem + s * STAGE_BYTES + h * (W_BYTES / 2) + row * 128;
                    uint32_t p[3][PART_COLS];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {                     // 16-byte pieces, where the 128-byte swizzle has put them
                        const float4 v = *reinterpret_cast<const float4*>(src + ((j ^ (row & 7)) << 4));
                        split_pair(v.x, v.y, p[0][2 * j], p[1][2 * j], p[2][2 * j]);
                        split_pair(v.z, v.w, p[0][2 * j + 1], p[1][2 * j + 1], p[2][2 * j + 1]);
                    }
                    const int pb = c % PARTS;
                    ok = __all_sync(0xffffffffu, tma::mbar_wait(&a_empty[pb], ((c / PARTS) & 1) ^ 1, abort_flag, status, 3));
                    if (!ok) break;
                    tc5::fence_after();
                    const uint32_t dst = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(2 * BN + pb * A_COLS);
#pragma unroll
                    for (int q = 0; q < 3; ++q) tc5::st16(dst + (uint32_t)(q * PART_COLS), p[q]);
                    tc5::wait_st();
                    tc5::fence_before();
                    tma::mbar_arrive(&a_full[pb]);
                    if (h == 1) tma::mbar_arrive(&empty[s]);
                }
            }
        }
    } else {
        const int row = (warp & 3) * 32 + lane, half = (warp - 6) >> 2;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * HALF);
        pdl_wait();
        int c = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < sh.items && ok; item += gridDim.x) {
            place(item, m0, n0, step0, n_steps, share);
            float acc[HALF];
#pragma unroll
            for (int j = 0; j < HALF; ++j) acc[j] = 0.f;
            for (int i = 0; i < 2 * n_steps; ++i, ++c) {
                const int ab = c & 1;
                ok = __all_sync(0xffffffffu, tma::mbar_wait(&acc_full[ab], (c >> 1) & 1, abort_flag, status, 5));
                if (!ok) break;
                tc5::fence_after();
#pragma unroll
                for (int j = 0; j < HALF; j += 16) {
                    uint32_t r[16];
                    tc5::ld16(lanes + (uint32_t)(ab * BN + j), r);
                    tc5::wait_ld();
#pragma unroll
                    for (int u = 0; u < 16; ++u) acc[j + u] += __uint_as_float(r[u]);
                }
                tc5::fence_before();
                tma::mbar_arrive(&acc_empty[ab]);
            }
            if (!ok) break;
            const int n = n0 + row;
            const bool shared_k = sh.shares > 1;
            const float b = !shared_k && bias != nullptr && n < sh.N ? bias[n] : 0.f;
            float* dst = shared_k ? partial + (size_t)share * sh.M * sh.N + n : out + n;
            const long long ld = shared_k ? sh.N : ldo;
            uint32_t again[(HALF + 31) / 32] = {};                   // the sums that are not finite
            if (n < sh.N) {
#pragma unroll
                for (int j = 0; j < HALF; ++j) {
                    const int m = m0 + half * HALF + j;
                    if (m >= sh.M) break;
                    float* p = dst + (size_t)m * ld;
                    if (fabsf(acc[j]) <= 3.402823466e38f) *p = !shared_k && accumulate ? *p + (acc[j] + b) : acc[j] + b;
                    else again[j / 32] |= 1u << (j % 32);
                }
            }
            uint32_t any = 0u;
#pragma unroll
            for (int g = 0; g < (HALF + 31) / 32; ++g) any |= again[g];
            if (__any_sync(0xffffffffu, any != 0u)) {
                const Again to = {x, w, shared_k ? partial + (size_t)share * sh.M * sh.N : out, ldx, ld, sh.M, sh.N, sh.K, step0 * STEP,
                                  min(sh.K, (step0 + n_steps) * STEP), !shared_k && accumulate, b};
#pragma unroll
                for (int g = 0; g < (HALF + 31) / 32; ++g) make_again(again[g], m0 + half * HALF + 32 * g, n0 + (warp & 3) * 32, to);
            }
        }
    }

    tc5::fence_before();
    __syncthreads();
    if (*abort_flag) {
        // a wait ran out: give copies and instructions in flight time to land before the memory goes away
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) { }
        __syncthreads();
    }
    if (warp == 1) {
        tc5::fence_after();
        tc5::dealloc(tmem, 512);
    }
}

// out (+)= the shares' sums in the order of K (+ bias)
__global__ void __launch_bounds__(256) finish_kernel(const float* partial, int shares, float* out, long long ldo, int accumulate,
                                                     const float* __restrict__ bias, int M, int N, int vec) {
    pdl_launch();
    pdl_wait();
    const size_t plane = (size_t)M * N;
    if (vec) {
        const int per_row = N / 4;
        for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < (size_t)M * per_row; i += (size_t)gridDim.x * 256) {
            const int m = (int)(i / per_row), n = (int)(i % per_row) * 4;
            const float* p = partial + (size_t)m * N + n;
            float4* o = reinterpret_cast<float4*>(out + (size_t)m * ldo + n);
            const float4 old = accumulate ? *o : make_float4(0.f, 0.f, 0.f, 0.f);
            float4 v = *reinterpret_cast<const float4*>(p);
#pragma unroll 4
            for (int s = 1; s < shares; ++s) {
                const float4 t = *reinterpret_cast<const float4*>(p + s * plane);
                v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
            }
            if (bias != nullptr) { v.x += bias[n]; v.y += bias[n + 1]; v.z += bias[n + 2]; v.w += bias[n + 3]; }
            if (accumulate) { v.x = old.x + v.x; v.y = old.y + v.y; v.z = old.z + v.z; v.w = old.w + v.w; }
            *o = v;
        }
        return;
    }
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < plane; i += (size_t)gridDim.x * 256) {
        const int m = (int)(i / N), n = (int)(i % N);
        float v = partial[i];
        for (int s = 1; s < shares; ++s) v += partial[s * plane + i];
        if (bias != nullptr) v += bias[n];
        float* o = out + (size_t)m * ldo + n;
        *o = accumulate ? *o + v : v;
    }
}

constexpr int TILES = 6;
constexpr float PAYS_BESIDE = 8.0f, PAYS_FROM = 28.0f;      // us: see gg_gemm_f32_parts_pays
const int TILE_BN[TILES] = {32, 64, 96, 128, 160, 192};

struct Plan {
    int tile, shares, steps;
};

// The tile and the shares of K with the least modelled time: rounds of 148 items, each its stages at the tile's measured rate and 2.5 us
// beside, and for shares the second kernel with its traffic.  (Measured, us a stage: 1.43 to 1.84 up to 160 rows, 2.0 at 192.)
Plan plan_for(int M, int N, int K, int force_tile, int force_shares, float* modelled = nullptr) {
    static const float step_us[TILES] = {1.44f, 1.5f, 1.5f, 1.6f, 1.7f, 1.95f};
    const int all = (K + STEP - 1) / STEP;
    const long long n_tiles = (N + ROWS - 1) / ROWS;
    Plan best = {0, 1, all};
    float least = 0.f;
    bool any = false;
    for (int t = 0; t < TILES; ++t) {
        if (force_tile >= 0 && t != force_tile) continue;
        const long long m_tiles = (M + TILE_BN[t] - 1) / TILE_BN[t];
        for (int s = 1; s <= 16 && s <= all; ++s) {
            if (force_shares > 0 && s != force_shares) continue;
            const int steps = (all + s - 1) / s;
            if ((all + steps - 1) / steps != s) continue;            // (a share would be empty)
            const long long rounds = (m_tiles * n_tiles * s + 147) / 148;
            float us = (float)rounds * ((float)steps * step_us[t] + 2.5f);
            if (s > 1) us += 3.0f + (float)(s + 1) * (float)M * (float)N * (4e-6f / 4.0f);
            if (!any || us < least) { best = {t, s, steps}; least = us; any = true; }
        }
    }
    if (modelled != nullptr) *modelled = least;
    return best;
}

template <int BN, int STAGES, int PARTS>
int launch_tile(const float* x, long long ldx, const float* w, float* out, long long ldo, int accumulate, const float* bias, float* partial,
                const bf16* parts, int ldp, Shape sh, int* status, cudaStream_t stream) {
    constexpr size_t smem = 1024 + (size_t)STAGES * (W_BYTES + 3 * BN * STEP * 2) + 8 * (3 * STAGES + 2 * PARTS + 4) + 16;
    static_assert(smem <= 227 * 1024, "shared memory");
    auto kern = parts_kernel<BN, STAGES, PARTS>;
    static int known[GG_MAX_DEVICES] = {};
    int resident = 0;
    int rc = gg_resident(kern, THREADS, smem, known, resident);
    if (rc != 0) return rc;
    sh.m_tiles = (sh.M + BN - 1) / BN;
    const long long items = (long long)sh.m_tiles * sh.n_tiles * sh.shares;
    if (items > 0x7fffffffLL || resident <= 0) return GG_ERR_ARG;
    sh.items = (int)items;
    CUtensorMap map_w, map_x;
    tma::EncodeTiledFn fn = tma::encode_fn();
    if (fn == nullptr) return GG_ERR_TMAP;
    cuuint64_t dims[2] = {(cuuint64_t)sh.K, (cuuint64_t)sh.N};
    cuuint64_t strides[1] = {(cuuint64_t)sh.K * 4};
    cuuint32_t box[2] = {32u, (cuuint32_t)ROWS}, estr[2] = {1, 1};
    if (fn(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return GG_ERR_TMAP;
    if ((rc = tma::make_map_bf16(&map_x, parts, 3ull * sh.M, sh.K, ldp, BN)) != 0) return rc;
    const int grid = sh.items < resident ? sh.items : resident;
    return gg_launch(kern, dim3(grid), dim3(THREADS), smem, stream, 1, map_w, map_x, x, ldx, w, out, ldo, accumulate, bias, partial, sh, status);
}

}  // namespace

static int parts_ld(int K) { return (K + 7) / 8 * 8; }

// Rows of x that are multiplied at a time: their parts are one and a half times x, so what they take is bounded by about 256 MB
// (a multiple of every tile's rows, 1,920 of them at least: 21 columns of tiles and more).
static int slab_rows(int K) {
    const long long rows = (256LL << 20) / (6LL * parts_ld(K)) / 1920 * 1920;
    return rows < 1920 ? 1920 : rows > 0x3fffffff ? 0x3fffffff / 1920 * 1920 : (int)rows;
}

static long long parts_bytes(int M, int K) { return (3LL * M * parts_ld(K) * 2 + 255) / 256 * 256; }

// Bytes of scratch that gg_gemm_f32_parts needs: the parts of a slab's rows, then the shares' sums.
GG_API gg_gemm_f32_parts_scratch(int M, int N, int K, int force_tile, int force_shares, long long* bytes) {
    if (M <= 0 || N <= 0 || K <= 0 || bytes == nullptr) return GG_ERR_ARG;
    const int slab = slab_rows(K);
    *bytes = 0;
    for (int m : {M < slab ? M : slab, M % slab}) {                  // (the last slab may be cut into shares where the others are not)
        if (m == 0) continue;
        const Plan p = plan_for(m, N, K, force_tile, force_shares);
        const long long need = parts_bytes(m, K) + (p.shares > 1 ? (long long)p.shares * m * N * 4 : 0);
        if (need > *bytes) *bytes = need;
    }
    return 0;
}

// Is a product of this size quicker in parts than on the CUDA cores?  On the GPU alone it is from 17 rows and K = 1,024 on (us, CUDA cores |
// parts: 17 rows by 2,048 x 2,048 21.9 | 13.8, 4,096 x 2,048 23.5 | 19.5; 64 rows 24.3 | 14.8, 46.4 | 20.2; 100 rows by 1,024 x 1,024 13.5 | 11.3,
// 512 x 512 7.3 | 8.1), but it is two or three launches instead of one, 4.5 us of the host's time each, and the host takes some
// 28 us for a product and what lies between it and the next (115 us a layer): a step of shorter products waits for the host whatever
// they are.  So the CUDA cores' time, modelled, has to be PAYS_FROM at least and PAYS_BESIDE longer than the parts'.  (Prompts through
// four layers, us, nothing in parts | as it is | everything: 1,024 wide, 17 tokens 490 | 478 | 523, 40 573 | 540 | 556, 100 796 | 555 | 594;
// 2,048 wide, 17 tokens 923 | 651 | 660, 100 1,983 | 717 | 847.)  Below K = 256 the sums are no more exact than theirs (K = 128: 1.1e-7 both).
GG_API gg_gemm_f32_parts_pays(int M, int N, int K, int* pays) {
    if (M <= 0 || N <= 0 || K <= 0 || pays == nullptr) return GG_ERR_ARG;
    *pays = 0;
    if (M < 17 || K < 256 || K % 4 != 0) return 0;
    // the CUDA cores' tiles as gemm_plain.cu chooses among them: rounds of 296, us per 1,000 of K, for up to 74, 148 and 296 tiles left
    static const float round_us[4][3] = {{7.5f, 10.5f, 11.4f}, {30, 30, 35}, {42, 42, 55}, {54, 54, 110}};
    static const int rows[4] = {32, 64, 64, 128}, cols[4] = {16, 32, 64, 64};
    float plain = 0.f;
    for (int i = 0; i < 4; ++i) {
        const long long t = (long long)((M + rows[i] - 1) / rows[i]) * ((N + cols[i] - 1) / cols[i]), left = t % 296;
        const float us = (round_us[i][2] * (float)(t / 296) + (left == 0 ? 0.f : round_us[i][left > 148 ? 2 : left > 74])) * (float)K * 1e-3f;
        if (i == 0 || us < plain) plain = us;
    }
    float parts = 0.f;
    plan_for(M, N, K, -1, 0, &parts);
    *pays = plain >= PAYS_FROM && parts + PAYS_BESIDE < plain;
    return 0;
}

// x[M, K] float32, rows ldx elements apart; w[N, K] float32 contiguous, on a 16-byte boundary, K a multiple of 4; out[M, N] float32, rows
// ldo apart; accumulate: out += product; bias (may be null): [N].  force_tile, force_shares: -1 and 0 for the plan (measurements
// and tests name them).
GG_API gg_gemm_f32_parts(const float* x, const float* w, float* out, int accumulate, int M, int N, int K, long long ldx, long long ldo,
                         const float* bias, void* scratch, long long scratch_bytes, int force_tile, int force_shares, int* status,
                         cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 != 0 || ldx < K || ldo < N || ((uintptr_t)w & 15) != 0 || scratch == nullptr || ((uintptr_t)scratch & 255) != 0)
        return GG_ERR_ARG;
    if (force_tile >= TILES) return GG_ERR_ARG;
    long long need = 0;
    gg_gemm_f32_parts_scratch(M, N, K, force_tile, force_shares, &need);
    if (scratch_bytes < need) return GG_ERR_ARG;
    const int ld = parts_ld(K), slab = slab_rows(K);
    bf16* parts = (bf16*)scratch;
    for (long long first = 0; first < M; first += slab, x += (size_t)slab * ldx, out += (size_t)slab * ldo) {
        const int m = (int)(M - first < slab ? M - first : slab);
        const Plan plan = plan_for(m, N, K, force_tile, force_shares);
        float* partial = (float*)((char*)scratch + parts_bytes(m, K));
        const long long quads = (long long)m * (K / 4);
        const int blocks = (int)((quads + 255) / 256 < 148 * 8 ? (quads + 255) / 256 : 148 * 8);
        int rc = gg_launch(split_rows_kernel, dim3(blocks), dim3(256), 0, stream, 1, x, ldx, parts, m, K, ld,
                           (int)(ldx % 4 == 0 && ((uintptr_t)x & 15) == 0));
        if (rc != 0) return rc;
        Shape sh = {m, N, K, 0, (N + ROWS - 1) / ROWS, plan.shares, plan.steps, 0};
#define GT(BN, ST, PA) rc = launch_tile<BN, ST, PA>(x, ldx, w, out, ldo, accumulate, bias, partial, parts, ld, sh, status, stream)
        switch (plan.tile) {
            case 0: GT(32, 4, 4); break;
            case 1: GT(64, 3, 4); break;
            case 2: GT(96, 3, 4); break;
            case 3: GT(128, 2, 4); break;
            case 4: GT(160, 2, 4); break;
            default: GT(192, 2, 2); break;
        }
#undef GT
        if (rc != 0) return rc;
        if (plan.shares == 1) continue;
        const int vec = N % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)out & 15) == 0;
        const long long n = (long long)m * (vec ? N / 4 : N);
        const int fb = (int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
        if ((rc = gg_launch(finish_kernel, dim3(fb), dim3(256), 0, stream, 1, (const float*)partial, plan.shares, out, ldo, accumulate, bias, m, N, vec)) != 0)
            return rc;
    }
    return 0;
}

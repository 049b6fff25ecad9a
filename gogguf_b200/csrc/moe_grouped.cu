// The routed experts' products on the tcgen05 tensor cores, all experts in one launch.
//
//   place:   the (token, choice) pairs in the order (expert, pair): place[p], the experts' row ranges offsets[E + 1] and the
//            pairs' input rows gathered in that order (times the weight where it sits on the input).
//   product: rows [offsets[e], offsets[e + 1]) of x times expert e's matrix.  GATED: w [E][2][N][K], out bfloat16 =
//            out_scale act(gate, up) (times the row's weight); else w [E][N][K], out float32.
//
// The ranges are read on the device, so nothing goes back to the host and a decode step can be captured.  A persistent
// grid walks over tiles of 128 rows x BN rows of the expert's matrix (gated: BN / 2 of gate and the BN / 2 of up that belong
// to them, so that the activation is applied to the accumulator); row tiles of one weight tile are neighbours in the
// walk and share it in L2.  Warp 0 loads (TMA, 128-byte swizzle), one thread of warp 1 multiplies into a double-buffered
// accumulator in tensor memory, warps 2 to 5 store.  A tile that is not full reads rows of the next expert and does not
// store them.
//
// What bounds it: with few rows per expert the weights' bytes (each touched expert's matrix is read once), with hundreds
// the tensor cores.  BN = 128 with two CTAs an SM for the first, BN = 256 for the second; see the rule at the launcher.  A
// stage holds as many rows of x as a tile can need (AROWS: the multiplication always reads 128, the others are what lies
// behind them in shared memory and end in rows that are not stored), so that with few pairs the ring is full of weights.
// Every mbarrier wait is bounded (tma_util.cuh).
#include "common.cuh"
#include "tma_util.cuh"

namespace {

constexpr int BM = 128, BK = 64, UMMA_K = 16, NUM_THREADS = 192, MAX_E = 1024;

__device__ __forceinline__ float clamped_glu(float g, float u, float limit, float slope, float up_offset) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-slope * g)) * (u + up_offset);
}

// ----------------------------------------------------------------------------- place and gather
// A block of 8 warps serves 8 pairs (or, behind the pairs' blocks, 8 of the E + 1 offsets): all threads walk over the P
// indices once and count for the 8 targets how many pairs come before them in the order (expert, pair), then warp w moves
// pair w's row.  No atomics, so the order is always the same; the indices (4 bytes a pair) stay in L2.  A choice without an
// expert (negative index) is filed behind the experts.
__global__ void __launch_bounds__(256) moe_place_gather_kernel(const bf16* h, const float* wts, const int* idx, int P, int E, int W,
                                                               int top, int weight_on_input, int* offsets, int* place,
                                                               float* row_wts, bf16* xs) {
    pdl_launch();
    pdl_wait();
    __shared__ int cnt[8][8];
    const int pair_blocks = (P + 7) / 8;
    const bool is_pairs = (int)blockIdx.x < pair_blocks;
    const int first = (is_pairs ? (int)blockIdx.x : (int)blockIdx.x - pair_blocks) * 8;
    int key[8], tie[8], c[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        c[j] = 0;
        if (is_pairs) {
            const int e = first + j < P ? idx[first + j] : -1;
            key[j] = e < 0 ? E : e;
            tie[j] = first + j;
        } else {
            key[j] = first + j;
            tie[j] = 0;
        }
    }
#pragma unroll 4
    for (int q = threadIdx.x; q < P; q += 256) {
        const int v = idx[q], e = v < 0 ? E : v;
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] += (e < key[j] || (e == key[j] && q < tie[j])) ? 1 : 0;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int s = __reduce_add_sync(0xffffffffu, c[j]);
        if (lane == 0) cnt[j][warp] = s;
    }
    __syncthreads();
    int at = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) at += cnt[warp][u];
    const int p = first + warp;
    if (!is_pairs) {
        if (lane == 0 && p <= E) offsets[p] = at;
        return;
    }
    if (p >= P) return;
    const float wt = wts[p];
    if (lane == 0) { place[p] = at; row_wts[at] = wt; }
    if (idx[p] < 0) return;                               // no product reads its row
    const uint4* src = reinterpret_cast<const uint4*>(h + (size_t)(p / top) * W);
    uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)at * W);
    for (int i0 = lane; i0 < W / 8; i0 += 4 * 32) {           // four loads, then four stores
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = src[min(i0 + 32 * k, W / 8 - 1)];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (weight_on_input) {
                __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&v[k]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float2 f = __bfloat1622float2(b[u]);
                    b[u] = __floats2bfloat162_rn(f.x * wt, f.y * wt);
                }
            }
            if (i0 + 32 * k < W / 8) dst[i0 + 32 * k] = v[k];
        }
    }
}

// ----------------------------------------------------------------------------- the products
template <int BN, int STAGES, int MINB, int AROWS>
__global__ void __launch_bounds__(NUM_THREADS, MINB) moe_grouped_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const int* offsets, int E,
    void* out, int N, int K, int gated, float limit, float slope, float up_offset, float out_scale, const float* row_wts,
    int* __restrict__ status) {
    constexpr int HALF = BN / 2;
    constexpr int A_BYTES = AROWS * BK * 2, STAGE_BYTES = A_BYTES + BN * BK * 2;
    static_assert(A_BYTES % 1024 == 0 && STAGE_BYTES >= BM * BK * 2, "the last stage's 128 rows end inside it");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;       // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2]
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    int* off = (int*)(tmem_slot + 4);          // [E + 1] first row of every expert
    int* start = off + E + 1;                  // [E + 1] first tile of every expert

    pdl_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_kb = (K + BK - 1) / BK;
    const int feat = gated ? HALF : BN;        // output columns of a tile
    const int tiles_n = (N + feat - 1) / feat;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { tma::mbar_init(&full[s], 1); tma::mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { tma::mbar_init(&acc_full[b], 1); tma::mbar_init(&acc_empty[b], 128); }
        *abort_flag = 0;
        tma::mbar_fence_init();
        tma::prefetch_map(&tmA);
        tma::prefetch_map(&tmB);
    }
    if (warp == 1) tc5::alloc(tmem_slot, 2 * BN);
    pdl_wait();
    for (int e = threadIdx.x; e <= E; e += NUM_THREADS) off[e] = offsets[e];
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    if (warp == 0) {                           // running sums of the experts' tile counts
        auto tiles_of = [&](int e) { return (off[e + 1] - off[e] + BM - 1) / BM * tiles_n; };
        auto scan = [&](int v) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += y;
            }
            return v;
        };
        if (E <= 32) {
            const int mine = lane < E ? tiles_of(lane) : 0, v = scan(mine);
            if (lane < E) start[lane] = v - mine;
            if (lane == 31) start[E] = v;
        } else {           // a run of neighbouring experts a lane (an odd number: no bank twice)
            const int per = (E + 31) / 32 | 1, e0 = min(E, lane * per), e1 = min(E, e0 + per);
            int mine = 0;
            for (int e = e0; e < e1; ++e) mine += tiles_of(e);
            int at = scan(mine);
            if (lane == 31) start[E] = at;
            at -= mine;
            for (int e = e0; e < e1; ++e) { start[e] = at; at += tiles_of(e); }
        }
    }
    __syncthreads();
    const uint32_t tmem_base = *tmem_slot;
    const int total = start[E];
    // the walk's tile t -> expert (the last that starts at or before t), row tile, column tile.  With many experts by halves: a walk
    // from one to the next took most of the 80 us of a layer with 1,000.
    auto tile_of = [&](int t, int& e, int& row0, int& rows, int& tn) {
        if (E > 32 && t >= start[e + 1]) {
            int hi = E;                                // start[++e] <= t < start[hi]
            ++e;
            while (hi - e > 1) {
                const int mid = (e + hi) >> 1;
                if (start[mid] <= t) e = mid; else hi = mid;
            }
        }
        while (t >= start[e + 1]) ++e;
        const int cnt = off[e + 1] - off[e], mt = (cnt + BM - 1) / BM, r = t - start[e];
        const int tm = r % mt;
        tn = r / mt;
        row0 = off[e] + tm * BM;
        rows = min(BM, cnt - tm * BM);
    };

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t tx = (uint32_t)STAGE_BYTES;
            int it = 0, e = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
                int row0, rows, tn;
                tile_of(t, e, row0, rows, tn);
                const int b0 = gated ? e * 2 * N + tn * HALF : e * N + tn * BN;
                const int b1 = gated ? b0 + N : b0 + HALF;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!tma::mbar_wait(&empty[s], ((uint32_t)(it / STAGES) & 1u) ^ 1u, abort_flag, status, 1)) { ok = false; break; }
                    tma::mbar_expect_tx(&full[s], tx);
                    uint8_t* sa = smem + s * STAGE_BYTES;
                    tma::load_2d(sa + A_BYTES, &tmB, &full[s], kb * BK, b0);
                    tma::load_2d(sa + A_BYTES + HALF * BK * 2, &tmB, &full[s], kb * BK, b1);
                    tma::load_2d(sa, &tmA, &full[s], kb * BK, row0);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = tc5::idesc_bf16(BM, BN, 0);
            int it = 0, i = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x, ++i) {
                const int buf = i & 1;
                ok = tma::mbar_wait(&acc_empty[buf], ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag, status, 4);
                if (!ok) break;
                tc5::fence_after();
                const uint32_t tacc = tmem_base + (uint32_t)(buf * BN);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = tma::mbar_wait(&full[s], (uint32_t)(it / STAGES) & 1u, abort_flag, status, 2);
                    if (!ok) break;
                    tc5::fence_after();
                    const uint32_t sa = tma::smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t adesc = tc5::smem_desc(sa, 16, 1024), bdesc = tc5::smem_desc(sa + A_BYTES, 16, 1024);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) tc5::mma(tacc, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc5::commit(&empty[s]);
                }
                if (ok) tc5::commit(&acc_full[buf]);
            }
        }
    } else {
        const int q = warp & 3;
        const int row = q * 32 + lane;
        int i = 0, e = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++i) {
            int row0, rows, tn;
            tile_of(t, e, row0, rows, tn);
            const int buf = i & 1;
            const bool live = row < rows;
            const size_t gi = (size_t)(row0 + (live ? row : 0));
            const float f = gated ? out_scale * (row_wts != nullptr ? row_wts[gi] : 1.0f) : 1.0f;
            if (!tma::mbar_wait(&acc_full[buf], (uint32_t)(i >> 1) & 1u, abort_flag, status, 3)) break;
            tc5::fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN);
            if (q * 32 < rows) {
#pragma unroll 1
                for (int c0 = 0; c0 < feat; c0 += 16) {
                    const int n = tn * feat + c0;
                    if (n >= N) break;
                    uint32_t g[16];
                    tc5::ld16(taddr + (uint32_t)c0, g);
                    if (gated) {
                        uint32_t u[16];
                        tc5::ld16(taddr + (uint32_t)(HALF + c0), u);
                        tc5::wait_ld();
                        if (!live) continue;
                        bf16* op = (bf16*)out + gi * N + n;
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = clamped_glu(__uint_as_float(g[j]), __uint_as_float(u[j]), limit, slope, up_offset) * f;
                        if (n + 16 <= N && (((uintptr_t)op) & 15) == 0) {
                            uint32_t pk[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                                pk[j] = *reinterpret_cast<uint32_t*>(&h2);
                            }
                            reinterpret_cast<uint4*>(op)[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                            reinterpret_cast<uint4*>(op)[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (n + j < N) op[j] = __float2bfloat16_rn(v[j]);
                        }
                    } else {
                        tc5::wait_ld();
                        if (!live) continue;
                        float* op = (float*)out + gi * N + n;
                        if (n + 16 <= N && (((uintptr_t)op) & 15) == 0) {
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                reinterpret_cast<float4*>(op)[j] = make_float4(__uint_as_float(g[4 * j]), __uint_as_float(g[4 * j + 1]),
                                                                               __uint_as_float(g[4 * j + 2]), __uint_as_float(g[4 * j + 3]));
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (n + j < N) op[j] = __uint_as_float(g[j]);
                        }
                    }
                }
            }
            tc5::fence_before();
            tma::mbar_arrive(&acc_empty[buf]);       // 128 arrivals free the accumulator for the tile after next
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
        tc5::dealloc(tmem_base, 2 * BN);
    }
}

template <int BN, int STAGES, int MINB, int AROWS>
int launch(const void* x, const CUtensorMap& tb, const int* offsets, int P, int E, void* out, int N, int K,
           int gated, float limit, float slope, float up_offset, float out_scale, const float* row_wts, int* status,
           cudaStream_t stream) {
    constexpr int fixed = STAGES * (AROWS + BN) * BK * 2 + 1024 + 256;
    const int smem = fixed + 8 * (E + 1);
    auto kern = moe_grouped_kernel<BN, STAGES, MINB, AROWS>;
    static bool configured = false;
    if (!configured) {
        cudaError_t er = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, fixed + 8 * (MAX_E + 1));
        if (er != cudaSuccess) return (int)er;
        configured = true;
    }
    CUtensorMap ta;
    const int rc = tma::make_map_bf16(&ta, x, (unsigned long long)P, K, K, AROWS);
    if (rc != 0) return rc;
    const int feat = gated ? BN / 2 : BN;
    const long long most = ((long long)(P < E ? P : E) + P / BM) * ((N + feat - 1) / feat);      // tiles, at most
    const int grid = (int)(most < 148LL * MINB ? most : 148LL * MINB);
    return gg_launch(kern, dim3(grid), dim3(NUM_THREADS), smem, stream, 1, ta, tb, offsets, E, out, N, K, gated, limit,
                     slope, up_offset, out_scale, row_wts, status);
}

}  // namespace

// idx[P] the pairs' experts (negative: none), h [P / top, W] bfloat16 (W a multiple of 8, 16-byte aligned rows), wts[P].
// offsets[E + 1], place[P], row_wts[P] (the weights in sorted order), xs [P, W].
GG_API gg_moe_place_gather(const void* h, const float* wts, const int* idx, int P, int E, int W, int top, int weight_on_input,
                           int* offsets, int* place, float* row_wts, void* xs, cudaStream_t stream) {
    if (P <= 0) return 0;
    if (E <= 0 || E > MAX_E || W <= 0 || (W % 8) || top <= 0 || P % top || (((uintptr_t)h | (uintptr_t)xs) & 15)) return GG_ERR_ARG;
    return gg_launch(moe_place_gather_kernel, dim3((P + 7) / 8 + (E + 8) / 8), dim3(256), 0, stream, 1, (const bf16*)h, wts, idx, P, E,
                     W, top, weight_on_input, offsets, place, row_wts, (bf16*)xs);
}

// x [P, K] rows in sorted order, of which expert e has offsets[e] .. offsets[e + 1].  row_wts (may be null; gated only): [P].
// status: one int on the device, zero unless a bounded wait ran out.
GG_API gg_moe_grouped(const void* x, const void* w, const int* offsets, int P, int E, void* out, int N, int K, int gated,
                      float limit, float slope, float up_offset, float out_scale, const float* row_wts, int* status,
                      cudaStream_t stream) {
    if (P <= 0) return 0;
    if (E <= 0 || E > MAX_E || N <= 0 || K <= 0 || (K % 8) || status == nullptr || (((uintptr_t)x | (uintptr_t)w) & 15) ||
        (long long)E * 2 * N > 0x7fffffffLL)
        return GG_ERR_ARG;
    // Measured, gate/up + down, us with 128-wide tiles / 256-wide ones by pairs per expert: 16 experts of 4,096 x 2,048: 32 147 / 147, 96 155 / 156,
    // 128 192 / 183, 160 263 / 214, 256 289 / 255, 512 477 / 420; 16 of 2,048 x 1,024: 32 44 / 48, 96 48 / 53, 128 68 / 68, 256 92 / 88,
    // 512 133 / 120; 64 of 2,048 x 768: 32 113 / 124, 96 128 / 135, 128 160 / 157.  (8 of 1,024 x 512 keep to the narrow tiles at any number:
    // 512 27 / 28.)  Few pairs: an expert may have all of them (the rows of a padded batch all go to the first), so P bounds the rows of a tile.
    const bool wide = P >= 128LL * E;
    CUtensorMap tb;
    const int rc = tma::make_map_bf16(&tb, w, (unsigned long long)E * (gated ? 2 : 1) * N, K, K, wide ? 128 : 64);
    if (rc != 0) return rc;
#define GG_MG(BN, ST, MINB, AR) return launch<BN, ST, MINB, AR>(x, tb, offsets, P, E, out, N, K, gated, limit, slope, up_offset, \
                                                                out_scale, row_wts, status, stream)
    if (wide) GG_MG(256, 4, 1, 128);
    if (P <= 16) GG_MG(128, 5, 2, 16);
    if (P <= 64) GG_MG(128, 4, 2, 64);
    GG_MG(128, 3, 2, 128);
#undef GG_MG
}

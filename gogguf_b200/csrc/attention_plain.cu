// Plain attention over the paged cache, for prefill and decode alike.
//
// One block per (token, query head).  The token at position p of sequence b sees the cached
// keys lo..p of that sequence (itself included: its key was written before this kernel runs),
// lo = 0, or p - window + 1 for a windowed layer, or the start of p's chunk of `chunk` positions (counted from the
// sequence's start), whichever is latest.  Query head h reads kv head h / (nq / nkv).
// Scores, the running maximum, the exponentials, their sum and the weighted sum of values are
// float32.  The values' head size dv may differ from the keys' d.  With `sink` (one float per query head), the
// softmax's denominator also holds exp(sink[h]): a score without a key or a value, not scaled.  `out_scale`
// multiplies the result (a mixer whose output is weighted takes the weight here, before any rounding), and so does
// sigmoid(gate[t, h dv + i]) where the layer has a gate per output element.
// This is the 32-bit path and the twin the fast kernels are checked against; it
// restates ops.AttentionScoresInto (pkg/ops/attention.go:10-47) and replaces the reference's
// attn_qk / softmax / attn_v PTX kernels (pkg/gpu/cuda/ptx.go:679-889), which the host loops
// over heads.
//
// What bounds it is latency: a key costs a table read, a row read and a reduction over the warp before its
// exponential is known.  So a warp takes eight neighbouring keys at a time (eight rows in flight, eight reductions side
// by side, one running maximum and one rescaling for the eight), and eight warps share a token's keys: a decode step has
// few (token, head) pairs.  Where even so most SMs would have nothing to do, up to eight blocks share a token's keys: they form a
// cluster, and each leaves its sums in the shared memory of the first, which adds them in the order of the shares.  A token's keys are
// cut by its position and the most shares of the step, which follow from the heads and the number of tokens rounded up to a power of two: a
// captured step's padding rows and wider tables change nothing.
#include <type_traits>
#include "common.cuh"

#define ATT_WARPS 8
#define ATT_KEYS 8
#define ATT_MAXD 256
#define ATT_SHARE_KEYS 128
#define ATT_SHARES 8                     // at most (the warps' factors and the shares' are kept in one array)

template <typename T> __device__ __forceinline__ float4 att_load4(const T* p);
template <> __device__ __forceinline__ float4 att_load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 att_load4<bf16>(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// NV > 0: d and dv are multiples of 4 up to 128 NV and the pools lie on 16-byte boundaries: a lane owns columns 4 lane .. + 3
// of every 128, and the keys and values of a warp's eight positions are all asked for at once, without a branch between
// the loads (with element loads behind `i < dv` the four groups of values waited for one another: 55 against 19 us for 4
// tokens, 16 heads of 128 and contexts around 600).  NV = 0: any sizes, element loads.
// SHARED: blockIdx.z is the block's share of the keys (its rank in the cluster) out of gridDim.z.  Few (token, head) pairs leave the chip
// idle and their keys a chain: 16 heads of 128, 1 token behind 4,000 keys 105 us in one share, now 22; 4 behind 900 26.5 | 13.2, 8 behind
// 900 42.5 | 20.9; 64 behind 900 fill it and stay as they were (125.5).
template <typename T, int NV, bool SHARED>
__global__ void __launch_bounds__(ATT_WARPS * 32) attention_plain_kernel(
    const T* q, const T* k_pool, const T* v_pool, T* __restrict__ out,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token,
    const int* __restrict__ page_table, int max_pages, int page_size,
    int nq, int nkv, int d, int dv, float scale, int window, int chunk, const float* __restrict__ sink, float out_scale,
    const T* gate, long long ldg, int most_shares, const PageBounds pb) {
    pdl_launch();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                       // [d]
    float* accs = sm + d;                 // [ATT_WARPS][dv]
    float* ml = accs + ATT_WARPS * dv;    // [ATT_WARPS][2]
    float* got = ml + 2 * ATT_WARPS;      // SHARED: the shares' sums, maxima and weights, [shares][dv + 2], in the first block
    const int share = SHARED ? (int)blockIdx.z : 0, launched = SHARED ? (int)gridDim.z : 1;
    const int t = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* o = out + ((size_t)t * nq + h) * dv;
    const int b = seq_of_token[t];
    if (b < 0) {
        if (share == 0)
            for (int i = threadIdx.x; i < dv; i += blockDim.x) o[i] = from_f<T>(0.f);
        return;
    }
    // (that the first block has started, so that its shared memory may be written to; waited for below)
    if (SHARED) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int pos = positions[t];
    const int g = h / (nq / nkv);
    int lo = 0;
    if (window > 0 && pos - window + 1 > 0) lo = pos - window + 1;
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    const T* qp = q + ((size_t)t * nq + h) * d;
    for (int i = threadIdx.x; i < d; i += blockDim.x) qs[i] = to_f<T>(qp[i]);
    __syncthreads();

    float acc[NV > 0 ? 4 * NV : ATT_MAXD / 32];
#pragma unroll
    for (int j = 0; j < (NV > 0 ? 4 * NV : ATT_MAXD / 32); ++j) acc[j] = 0.f;
    float m = -INFINITY, l = 0.f;
    const int* pt = page_table + (size_t)b * max_pages;
    float4 q4[NV > 0 ? NV : 1];
    bool in_k[NV > 0 ? NV : 1], in_v[NV > 0 ? NV : 1];
    if (NV > 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            in_k[c] = 128 * c + 4 * lane < d;
            in_v[c] = 128 * c + 4 * lane < dv;
            q4[c] = in_k[c] ? *reinterpret_cast<const float4*>(qs + 128 * c + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    // (a share of at least ATT_SHARE_KEYS keys; the blocks beyond a token's shares have none)
    const int shares = SHARED ? min(most_shares, 1 + (pos - lo) / ATT_SHARE_KEYS) : 1;
    for (int j0 = share < shares ? lo + (share * ATT_WARPS + warp) * ATT_KEYS : pos + 1; j0 <= pos; j0 += shares * ATT_WARPS * ATT_KEYS) {
        size_t base[ATT_KEYS];
        float dot[ATT_KEYS];
#pragma unroll
        for (int u = 0; u < ATT_KEYS; ++u) {
            const int j = min(j0 + u, pos);              // past the last key: its row again, with weight zero
            const int page = gg_page(pt, j / page_size, max_pages, pb, 41);
            base[u] = ((size_t)page * nkv + g) * page_size + (j % page_size);
            dot[u] = 0.f;
        }
        float4 v4[NV > 0 ? ATT_KEYS : 1][NV > 0 ? NV : 1];
        if (NV > 0) {
            float4 k4[ATT_KEYS][NV > 0 ? NV : 1];
#pragma unroll
            for (int u = 0; u < ATT_KEYS; ++u)
#pragma unroll
                for (int c = 0; c < NV; ++c) {           // (a lane beyond the row reads its first columns and drops them)
                    k4[u][c] = att_load4<T>(k_pool + base[u] * d + (in_k[c] ? 128 * c + 4 * lane : 0));
                    v4[u][c] = att_load4<T>(v_pool + base[u] * dv + (in_v[c] ? 128 * c + 4 * lane : 0));
                }
#pragma unroll
            for (int u = 0; u < ATT_KEYS; ++u)
#pragma unroll
                for (int c = 0; c < NV; ++c) {
                    const float r = fmaf(q4[c].w, k4[u][c].w, fmaf(q4[c].z, k4[u][c].z, fmaf(q4[c].y, k4[u][c].y, q4[c].x * k4[u][c].x)));
                    dot[u] += in_k[c] ? r : 0.f;
                }
        } else {
#pragma unroll 4
            for (int i = lane; i < d; i += 32) {
                const float qv = qs[i];
#pragma unroll
                for (int u = 0; u < ATT_KEYS; ++u) dot[u] = fmaf(qv, to_f<T>(k_pool[base[u] * d + i]), dot[u]);
            }
        }
        float mn = m;
#pragma unroll
        for (int u = 0; u < ATT_KEYS; ++u) {
            // (no branch: the eight reductions run side by side)
            const float r = warp_sum(dot[u]) * scale;
            dot[u] = j0 + u <= pos ? r : -INFINITY;
            mn = fmaxf(mn, dot[u]);
        }
        const float corr = expf(m - mn);
        l *= corr;
#pragma unroll
        for (int u = 0; u < ATT_KEYS; ++u) {
            dot[u] = j0 + u <= pos ? expf(dot[u] - mn) : 0.f;
            l += dot[u];
        }
        if (NV > 0) {
#pragma unroll
            for (int c = 0; c < NV; ++c) {
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[4 * c + e] *= corr;
#pragma unroll
                for (int u = 0; u < ATT_KEYS; ++u) {
                    const bool in = j0 + u <= pos;
                    acc[4 * c + 0] = fmaf(dot[u], in ? v4[u][c].x : 0.f, acc[4 * c + 0]);
                    acc[4 * c + 1] = fmaf(dot[u], in ? v4[u][c].y : 0.f, acc[4 * c + 1]);
                    acc[4 * c + 2] = fmaf(dot[u], in ? v4[u][c].z : 0.f, acc[4 * c + 2]);
                    acc[4 * c + 3] = fmaf(dot[u], in ? v4[u][c].w : 0.f, acc[4 * c + 3]);
                }
            }
        } else
#pragma unroll
        for (int jj = 0; jj < ATT_MAXD / 32; ++jj) {
            const int i = lane + 32 * jj;
            if (i < dv) {
                float v[ATT_KEYS];
#pragma unroll
                for (int u = 0; u < ATT_KEYS; ++u) v[u] = to_f<T>(v_pool[base[u] * dv + i]);
                float& o = acc[NV > 0 ? 0 : jj];
                o *= corr;
#pragma unroll
                for (int u = 0; u < ATT_KEYS; ++u) o = fmaf(dot[u], j0 + u <= pos ? v[u] : 0.f, o);
            }
        }
        m = mn;
    }
    if (NV > 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c)
            if (in_v[c])
                *reinterpret_cast<float4*>(accs + warp * dv + 128 * c + 4 * lane) = make_float4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
    } else {
#pragma unroll
        for (int jj = 0; jj < ATT_MAXD / 32; ++jj) {
            const int i = lane + 32 * jj;
            if (i < dv) accs[warp * dv + i] = acc[NV > 0 ? 0 : jj];
        }
    }
    if (lane == 0) { ml[warp * 2] = m; ml[warp * 2 + 1] = l; }
    __syncthreads();
    if (SHARED) {
        float M = -INFINITY, L = 0.f, f[ATT_WARPS];
        for (int w = 0; w < ATT_WARPS; ++w) M = fmaxf(M, ml[w * 2]);
        for (int w = 0; w < ATT_WARPS; ++w) { f[w] = ml[w * 2] == -INFINITY ? 0.f : expf(ml[w * 2] - M); L += ml[w * 2 + 1] * f[w]; }
        uint32_t first;
        asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(first) : "r"((uint32_t)__cvta_generic_to_shared(got + share * (dv + 2))));
        auto put = [&](int i, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(first + 4u * (uint32_t)i), "f"(v) : "memory"); };
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        for (int i = threadIdx.x; i < dv; i += blockDim.x) {
            float s = 0.f;
            for (int w = 0; w < ATT_WARPS; ++w) s += accs[w * dv + i] * f[w];
            put(i, s);
        }
        if (threadIdx.x == 0) { put(dv, M); put(dv + 1, L); }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (share > 0) return;
        M = sink != nullptr ? sink[h] : -INFINITY;
        for (int r = 0; r < launched; ++r) M = fmaxf(M, got[r * (dv + 2) + dv]);
        L = sink != nullptr ? expf(sink[h] - M) : 0.f;
        for (int r = 0; r < launched; ++r) {
            const float mr = got[r * (dv + 2) + dv];
            f[r] = mr == -INFINITY ? 0.f : expf(mr - M);
            L += got[r * (dv + 2) + dv + 1] * f[r];
        }
        const float inv = out_scale / L;
        for (int i = threadIdx.x; i < dv; i += blockDim.x) {
            float s = 0.f;
            for (int r = 0; r < launched; ++r) s += got[r * (dv + 2) + i] * f[r];
            s *= inv;
            if (gate != nullptr) s /= 1.0f + expf(-to_f<T>(gate[(size_t)t * ldg + (size_t)h * dv + i]));
            o[i] = from_f<T>(s);
        }
        return;
    }
    float M = sink != nullptr ? sink[h] : -INFINITY;
    for (int w = 0; w < ATT_WARPS; ++w) M = fmaxf(M, ml[w * 2]);
    float L = sink != nullptr ? expf(sink[h] - M) : 0.f;
    float f[ATT_WARPS];
    for (int w = 0; w < ATT_WARPS; ++w) { f[w] = ml[w * 2] == -INFINITY ? 0.f : expf(ml[w * 2] - M); L += ml[w * 2 + 1] * f[w]; }
    const float inv = out_scale / L;
    for (int i = threadIdx.x; i < dv; i += blockDim.x) {
        float s = 0.f;
        for (int w = 0; w < ATT_WARPS; ++w) s += accs[w * dv + i] * f[w];
        s *= inv;
        if (gate != nullptr) s /= 1.0f + expf(-to_f<T>(gate[(size_t)t * ldg + (size_t)h * dv + i]));
        o[i] = from_f<T>(s);
    }
}

// ----------------------------------------------------------------------------- prompts in 32 bits
// The same attention for steps that bring many tokens a sequence, float32, d and dv multiples of 4 up to 128, pools on 16-byte
// boundaries.  A block takes 32 consecutive (token, head) rows of one sequence and one kv head (tokens slowest, the heads that share the
// kv head fastest) and walks over the keys that any of them sees, 32 at a time in two stages of shared memory, so a key is read
// once for 32 rows where attention_plain_kernel reads it for each.  128 threads: thread (tx, ty) has the scores of rows ty and ty + 16
// with keys tx, tx + 8, .. and, of the same rows, the output's columns 4 tx .. + 3 of every 32; a row's maximum and sum are its
// eight threads' (neighbouring lanes).  Rows of shared memory are padded by four floats: a read of eight rows touches every bank once.
// Multiply-adds bound it (a score and a value product each, 16 bytes of shared memory to some five of them).  One prompt of 450 tokens, 16
// heads of 128 over 8 kv heads: 215 us a row at a time, 141 in tiles; 16 tokens behind 4,000 keys, eight tiles of 126 steps each: 191 and 934.
#define APT_ROWS 32
#define APT_KEYS 32
#define APT_P (APT_KEYS + 4)

__device__ __forceinline__ void apt_cp16(float* smem, const float* gmem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem) : "memory");
}

__global__ void __launch_bounds__(128) attention_plain_tile_kernel(
    const float* q, const float* k_pool, const float* v_pool, float* __restrict__ out, const int* __restrict__ positions,
    const int* __restrict__ seq_of_token, const int* __restrict__ cu_seqlens, int n_seqs, const int* __restrict__ page_table, int max_pages,
    int page_size, int nq, int nkv, int d, int dv, float scale, int window, int chunk, const float* __restrict__ sink, float out_scale,
    const float* gate, long long ldg, int early_release, const PageBounds pb) {
    if (early_release) pdl_launch();              // (the grid is resident as a whole; the note on dependent launches in common.cuh)
    extern __shared__ __align__(16) float sm[];
    const int LD = d + 4, LV = dv + 4, G = nq / nkv, g = blockIdx.y;
    float* qs = sm;                               // [32][LD]
    float* ks = qs + APT_ROWS * LD;               // [2][32][LD]
    float* vs = ks + 2 * APT_KEYS * LD;           // [2][32][LV]
    float* ps = vs + 2 * APT_KEYS * LV;           // [32][APT_P]
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    int b = 0, tile = blockIdx.x, t0 = 0, n_new = 0;
    for (; b < n_seqs; ++b) {
        t0 = cu_seqlens[b];
        n_new = cu_seqlens[b + 1] - t0;
        const int tiles = (n_new * G + APT_ROWS - 1) / APT_ROWS;
        if (tile < tiles) break;
        tile -= tiles;
    }
    if (b >= n_seqs) return;
    pdl_wait();
    const int f0 = tile * APT_ROWS, rows = min(APT_ROWS, n_new * G - f0);
    b = seq_of_token[t0];
    if (b < 0) {                                  // a padding sequence: zero rows
        for (int i = tid; i < rows * dv; i += 128) {
            const int f = f0 + i / dv;
            out[((size_t)(t0 + f / G) * nq + g * G + f % G) * dv + i % dv] = 0.f;
        }
        return;
    }
    const int tl0 = f0 / G, tl1 = (f0 + rows - 1) / G, pos0 = positions[t0 + tl0], last = pos0 + (tl1 - tl0);
    auto first_key = [&](int pos) {
        const int lo = window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0;
        return chunk > 0 ? max(lo, pos / chunk * chunk) : lo;
    };
    const int lo = first_key(pos0);               // (no row's first key lies before that of the row before it)
    const int n_tiles = (last - lo) / APT_KEYS + 1;
    const int* pt = page_table + (size_t)b * max_pages;
    const int dc = d / 4, vc = dv / 4;
    auto load = [&](int it) {
        if (it < n_tiles) {
            float* kd = ks + (it & 1) * APT_KEYS * LD;
            float* vd = vs + (it & 1) * APT_KEYS * LV;
            const int rr = tid >> 2, part = tid & 3;                     // four threads a row
            const int j = min(lo + it * APT_KEYS + rr, last);            // past the last key: its row again, with weight zero
            const int page = gg_page(pt, j / page_size, max_pages, pb, 41);
            const size_t at = ((size_t)page * nkv + g) * page_size + (j % page_size);
            for (int c = part; c < dc; c += 4) apt_cp16(kd + rr * LD + 4 * c, k_pool + at * d + 4 * c);
            for (int c = part; c < vc; c += 4) apt_cp16(vd + rr * LV + 4 * c, v_pool + at * dv + 4 * c);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    {
        const int rr = tid >> 2, part = tid & 3, f = f0 + min(rr, rows - 1);
        const float* src = q + ((size_t)(t0 + f / G) * nq + g * G + f % G) * d;
        for (int c = part; c < dc; c += 4) apt_cp16(qs + rr * LD + 4 * c, src + 4 * c);
    }
    load(0);
    float acc[2][4][4], m[2], l[2];
    int pos[2], low[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int f = f0 + min(ty + 16 * i, rows - 1);
        pos[i] = pos0 + (f / G - tl0);
        low[i] = first_key(pos[i]);
        m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][c][e] = 0.f;
    }
#pragma unroll 1
    for (int it = 0; it < n_tiles; ++it) {
        load(it + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float* kt = ks + (it & 1) * APT_KEYS * LD;
        const float* vt = vs + (it & 1) * APT_KEYS * LV;
        float s[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int c = 0; c < dc; ++c) {
            float4 a[2], k4[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (ty + 16 * i) * LD + 4 * c);
#pragma unroll
            for (int j = 0; j < 4; ++j) k4[j] = *reinterpret_cast<const float4*>(kt + (tx + 8 * j) * LD + 4 * c);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = fmaf(a[i].w, k4[j].w, fmaf(a[i].z, k4[j].z, fmaf(a[i].y, k4[j].y, fmaf(a[i].x, k4[j].x, s[i][j]))));
        }
        const int j0 = lo + it * APT_KEYS + tx;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float mn = m[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int at = j0 + 8 * j;
                s[i][j] = at <= pos[i] && at >= low[i] ? s[i][j] * scale : -INFINITY;
                mn = fmaxf(mn, s[i][j]);
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            const float use = mn == -INFINITY ? 0.f : mn, corr = expf(m[i] - use);       // (0 while the row has seen nothing)
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = expf(s[i][j] - use);
                sum += p;
                ps[(ty + 16 * i) * APT_P + tx + 8 * j] = p;
            }
            l[i] = l[i] * corr + sum;                                                    // this thread's keys; added up at the end
            m[i] = mn;
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][c][e] *= corr;
        }
        __syncwarp();                                                    // a row's weights are its own warp's
        // Keys that one row sees and another does not lie in tiles on an edge: there a value that a row does not see is not
        // multiplied (it may be an infinity, and its weight is zero).
        const int from = lo + it * APT_KEYS;
        auto values = [&](auto edge) {
#pragma unroll 2
            for (int k0 = 0; k0 < APT_KEYS; k0 += 4) {
                float p[2][4];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float4 t = *reinterpret_cast<const float4*>(ps + (ty + 16 * i) * APT_P + k0);
                    p[i][0] = t.x; p[i][1] = t.y; p[i][2] = t.z; p[i][3] = t.w;
                }
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (4 * tx + 32 * c < dv) {
                            const float4 v = *reinterpret_cast<const float4*>(vt + (k0 + kk) * LV + 4 * tx + 32 * c);
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const int at = from + k0 + kk;
                                const bool in = !decltype(edge)::value || (at <= pos[i] && at >= low[i]);
                                acc[i][c][0] = fmaf(p[i][kk], in ? v.x : 0.f, acc[i][c][0]);
                                acc[i][c][1] = fmaf(p[i][kk], in ? v.y : 0.f, acc[i][c][1]);
                                acc[i][c][2] = fmaf(p[i][kk], in ? v.z : 0.f, acc[i][c][2]);
                                acc[i][c][3] = fmaf(p[i][kk], in ? v.w : 0.f, acc[i][c][3]);
                            }
                        }
                    }
            }
        };
        if (from + APT_KEYS - 1 > pos0 || from < first_key(last)) values(std::true_type{});
        else values(std::false_type{});
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int rr = ty + 16 * i, f = f0 + rr;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
        if (rr >= rows) continue;
        const int t = t0 + f / G, h = g * G + f % G;
        float factor = 1.f, L = l[i];
        if (sink != nullptr) {
            const float M = fmaxf(m[i], sink[h]);
            factor = expf(m[i] - M);
            L = L * factor + expf(sink[h] - M);
        }
        factor *= out_scale / L;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int col = 4 * tx + 32 * c;
            if (col >= dv) continue;
            float r[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                r[e] = acc[i][c][e] * factor;
                if (gate != nullptr) r[e] /= 1.0f + expf(-gate[(size_t)t * ldg + (size_t)h * dv + col + e]);
            }
            *reinterpret_cast<float4*>(out + ((size_t)t * nq + h) * dv + col) = make_float4(r[0], r[1], r[2], r[3]);
        }
    }
}

// q[T, nq, d] and out[T, nq, dv] in `dtype`; pools k [page][nkv][page_size][d], v [page][nkv][page_size][dv] in
// `dtype`, n_pages of them.  sink: null or one float per query head.
// gate: null or logits in `dtype`, rows ldg apart.  chunk 0: none.
// cu_seqlens (may be null): [n_seqs + 1] prefix sums of the step's tokens by sequence, a sequence's tokens at consecutive positions; with
// it, steps of 16 or more tokens a sequence on average take the tiled kernel where the sizes allow it: callers pass it where the tiles are
// quicker (kernels.py, attention_tiles_pay).
// status (may be null): where the debug build records a page id or table index out of range (code 41).
GG_API gg_attention_plain(const void* q, const void* k_pool, const void* v_pool, void* out, int dtype,
                          const int* positions, const int* seq_of_token, const int* page_table,
                          int max_pages, int page_size, int n_pages, int ntok, int nq, int nkv, int d, int dv,
                          float scale, int window, int chunk, const float* sink, float out_scale, const void* gate,
                          long long ldg, const int* cu_seqlens, int n_seqs, int* status, cudaStream_t stream) {
    if (ntok <= 0) return 0;
    if (d <= 0 || dv <= 0 || dv > ATT_MAXD || d > 4096 || nq <= 0 || nkv <= 0 || nq % nkv || nq > 65535 || page_size <= 0) return GG_ERR_ARG;
    // Tiles of 32 rows where most have 32 and the caller asks for them.
    if (cu_seqlens != nullptr && n_seqs > 0 && ntok >= 16LL * n_seqs && dtype == GG_F32 && d % 4 == 0 && dv % 4 == 0 && d <= 128 && dv <= 128 &&
        nkv <= 65535 && (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out) & 15) == 0) {
        const size_t tile_smem = (size_t)(APT_ROWS * (d + 4) + 2 * APT_KEYS * (d + 4 + dv + 4) + APT_ROWS * APT_P) * sizeof(float);
        static int known[GG_MAX_DEVICES] = {};
        int resident = 0;
        const int rc = gg_resident(attention_plain_tile_kernel, 128, 96 * 1024, known, resident);
        if (rc != 0) return rc;
        const long long tiles = ((long long)ntok * (nq / nkv) + APT_ROWS - 1) / APT_ROWS + n_seqs;
        if (tiles > 0x7fffffffLL) return GG_ERR_ARG;
        return gg_launch(attention_plain_tile_kernel, dim3((unsigned)tiles, nkv), dim3(128), tile_smem, stream, 1, (const float*)q,
                         (const float*)k_pool, (const float*)v_pool, (float*)out, positions, seq_of_token, cu_seqlens, n_seqs, page_table, max_pages,
                         page_size, nq, nkv, d, dv, scale, window, chunk, sink, out_scale, (const float*)gate, ldg,
                         tiles * nkv <= resident ? 1 : 0, PageBounds{n_pages, status});
    }
    // The most shares of a token's keys: as many as keep the grid within three blocks an SM; launched are no more than a token of the widest
    // context that the tables have room for would take.
    long long tokens = 1;
    while (tokens < ntok) tokens *= 2;
    int most = 1, shares = 1;
    while (most < ATT_SHARES && tokens * nq * most * 2 <= 148 * 3) most *= 2;
    while (shares < most && 1 + ((long long)max_pages * page_size - 1) / ATT_SHARE_KEYS > shares) shares *= 2;
    size_t smem = ((size_t)d + (size_t)ATT_WARPS * dv + 2 * ATT_WARPS) * sizeof(float);
    if (shares > 1) smem += (size_t)shares * (dv + 2) * sizeof(float);
    dim3 grid(ntok, nq, shares);
    // (the lanes' float4s: q and the warps' sums start on multiples of 16 bytes in shared memory when d and dv are multiples of 4)
    const int wide = d > dv ? d : dv;
    const int nv = (d % 4 == 0 && dv % 4 == 0 && wide <= 256 && (((uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0) ? (wide + 127) / 128 : 0;
#define GG_ATT_AS(NV, SH) return gg_launch(attention_plain_kernel<T, NV, SH>, grid, dim3(ATT_WARPS * 32), smem, stream, shares, \
            (const T*)q, (const T*)k_pool, (const T*)v_pool, (T*)out, positions, seq_of_token, page_table, \
            max_pages, page_size, nq, nkv, d, dv, scale, window, chunk, sink, out_scale, (const T*)gate, ldg, most, PageBounds{n_pages, status})
#define GG_ATT(NV) { if (shares > 1) GG_ATT_AS(NV, true); GG_ATT_AS(NV, false); }
    GG_DISPATCH_DTYPE(dtype, T,
        if (nv == 1) GG_ATT(1)
        if (nv == 2) GG_ATT(2)
        GG_ATT(0));
#undef GG_ATT
#undef GG_ATT_AS
}

// 1 if this library was built with checked page tables (the debug build), else 0.
GG_API gg_attention_plain_checked() { return gg_debug_bounds(); }

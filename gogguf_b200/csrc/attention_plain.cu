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
// few (token, head) pairs.  Keys are given out by position alone, so the result does not depend on the batch.
#include "common.cuh"

#define ATT_WARPS 8
#define ATT_KEYS 8
#define ATT_MAXD 256

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
template <typename T, int NV>
__global__ void __launch_bounds__(ATT_WARPS * 32) attention_plain_kernel(
    const T* q, const T* k_pool, const T* v_pool, T* __restrict__ out,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token,
    const int* __restrict__ page_table, int max_pages, int page_size,
    int nq, int nkv, int d, int dv, float scale, int window, int chunk, const float* __restrict__ sink, float out_scale,
    const T* gate, long long ldg, const PageBounds pb) {
    pdl_launch();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                       // [d]
    float* accs = sm + d;                 // [ATT_WARPS][dv]
    float* ml = accs + ATT_WARPS * dv;    // [ATT_WARPS][2]
    const int t = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* o = out + ((size_t)t * nq + h) * dv;
    const int b = seq_of_token[t];
    if (b < 0) {
        for (int i = threadIdx.x; i < dv; i += blockDim.x) o[i] = from_f<T>(0.f);
        return;
    }
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
    for (int j0 = lo + warp * ATT_KEYS; j0 <= pos; j0 += ATT_WARPS * ATT_KEYS) {
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

// q[T, nq, d] and out[T, nq, dv] in `dtype`; pools k [page][nkv][page_size][d], v [page][nkv][page_size][dv] in
// `dtype`, n_pages of them.  sink: null or one float per query head.
// gate: null or logits in `dtype`, rows ldg apart.  chunk 0: none.
// status (may be null): where the debug build records a page id or table index out of range (code 41).
GG_API gg_attention_plain(const void* q, const void* k_pool, const void* v_pool, void* out, int dtype,
                          const int* positions, const int* seq_of_token, const int* page_table,
                          int max_pages, int page_size, int n_pages, int ntok, int nq, int nkv, int d, int dv,
                          float scale, int window, int chunk, const float* sink, float out_scale, const void* gate,
                          long long ldg, int* status, cudaStream_t stream) {
    if (ntok <= 0) return 0;
    if (d <= 0 || dv <= 0 || dv > ATT_MAXD || d > 4096 || nq <= 0 || nkv <= 0 || nq % nkv || nq > 65535 || page_size <= 0) return GG_ERR_ARG;
    const size_t smem = ((size_t)d + (size_t)ATT_WARPS * dv + 2 * ATT_WARPS) * sizeof(float);
    dim3 grid(ntok, nq);
    // (the lanes' float4s: q and the warps' sums start on multiples of 16 bytes in shared memory when d and dv are multiples of 4)
    const int wide = d > dv ? d : dv;
    const int nv = (d % 4 == 0 && dv % 4 == 0 && wide <= 256 && (((uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0) ? (wide + 127) / 128 : 0;
#define GG_ATT(NV) return gg_launch(attention_plain_kernel<T, NV>, dim3(grid), dim3(ATT_WARPS * 32), smem, stream, 1, \
            (const T*)q, (const T*)k_pool, (const T*)v_pool, (T*)out, positions, seq_of_token, page_table, \
            max_pages, page_size, nq, nkv, d, dv, scale, window, chunk, sink, out_scale, (const T*)gate, ldg, PageBounds{n_pages, status})
    GG_DISPATCH_DTYPE(dtype, T,
        if (nv == 1) GG_ATT(1);
        if (nv == 2) GG_ATT(2);
        GG_ATT(0));
#undef GG_ATT
}

// 1 if this library was built with checked page tables (the debug build), else 0.
GG_API gg_attention_plain_checked() { return gg_debug_bounds(); }

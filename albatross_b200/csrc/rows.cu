// Row-wise glue of the batched path: embedding gather, layer norm, token-shift lerps.
//
// Restates, for [B,T,D] activations, reference/rwkv7.py:195 (embedding gather), :203/:213/:219
// (layer norms) and :280-281 / :319-320 (token shift + lerps). One block per row; fp16 in and
// out with the reference's rounding points (each torch op on an fp16 tensor rounds once).
#include "rows.cuh"

namespace ab {

namespace {

constexpr int RT = 256;

__device__ __forceinline__ float block_sum_rt(float v, float* red) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < RT / 32; ++i) t += red[i];
    return t;
}

// Row of the table that an id names; an id outside of it is clamped and reported, never followed.
__device__ __forceinline__ size_t token_row(int tok, int vocab) {
    if ((unsigned)tok >= (unsigned)vocab) {
        tok = tok < 0 ? 0 : vocab - 1;
        if (threadIdx.x == 0) atomicOr(&g_device_status, DEV_BAD_TOKEN);
    }
    return (size_t)tok;
}

__global__ void __launch_bounds__(RT) gather_rows_kernel(const __half* __restrict__ table, const int* __restrict__ idx,
                                                         int D, int vocab, __half* __restrict__ out) {
    const size_t m = blockIdx.x;
    const size_t tok = token_row(idx[m], vocab);
    const uint4* src = reinterpret_cast<const uint4*>(table + tok * D);
    uint4* dst = reinterpret_cast<uint4*>(out + m * D);
    for (int i = threadIdx.x; i < D / 8; i += RT)
        if (AB_BC(tok < (size_t)vocab && (i + 1) * 8 <= D)) dst[i] = src[i];
}

// out[m] = LN(x[src_row(m)]) with src_row = m * stride + offset (stride/offset pick last tokens).
__global__ void __launch_bounds__(RT) ln_rows_kernel(const __half* __restrict__ x, const __half* __restrict__ w,
                                                     const __half* __restrict__ b, int D, int stride, int offset,
                                                     __half* __restrict__ out) {
    __shared__ float red[RT / 32];
    const size_t m = blockIdx.x;
    const __half* xr = x + (m * stride + offset) * D;
    float s = 0.f;
    for (int i = threadIdx.x; i < D; i += RT) s += __half2float(xr[i]);
    const float mean = block_sum_rt(s, red) / (float)D;
    float q = 0.f;
    for (int i = threadIdx.x; i < D; i += RT) {
        const float d = __half2float(xr[i]) - mean;
        q += d * d;
    }
    const float rstd = rsqrtf(block_sum_rt(q, red) / (float)D + 1e-5f);
    for (int i = threadIdx.x; i < D; i += RT)
        out[m * D + i] = __float2half_rn((__half2float(xr[i]) - mean) * rstd * __half2float(w[i]) + __half2float(b[i]));
}

// The same with the row in registers, 16 bytes at a time, for the norm in front of the vocabulary head: its weights are requested
// while the preceding kernel still runs, and the product behind it may start its weights. Together with the first block's
// norm reading the embedding itself (token_row), two blocks of the network, 4096 wide: 8 sequences one step 176.7 -> 173.9 us, 64
// sequences 279.0 -> 276.5, 5 prompts of 37 tokens 350.4 -> 348.3.
constexpr int LV_MAXV = 4;
__global__ void __launch_bounds__(RT) ln_vec_kernel(const __half* __restrict__ x, const __half* __restrict__ w, const __half* __restrict__ b,
                                                    int D, int stride, int offset, __half* __restrict__ out, int use_pdl) {
    __shared__ float red[RT / 32];
    const size_t m = blockIdx.x;
    const int nv = D / 8;
    const uint4* xr = reinterpret_cast<const uint4*>(x + (m * stride + offset) * D);
    uint4 raw[LV_MAXV], wv[LV_MAXV], bv[LV_MAXV];
    if (use_pdl) pdl_launch_dependents();
#pragma unroll
    for (int v = 0; v < LV_MAXV; ++v) {
        const int i = threadIdx.x + v * RT;
        if (i < nv) {
            wv[v] = reinterpret_cast<const uint4*>(w)[i];
            bv[v] = reinterpret_cast<const uint4*>(b)[i];
        }
    }
    if (use_pdl) pdl_wait();
    float s = 0.f;
#pragma unroll
    for (int v = 0; v < LV_MAXV; ++v) {
        const int i = threadIdx.x + v * RT;
        if (i < nv) {
            // an ordinary (coherent) load that stays behind the wait above: the row was written by the preceding kernel
            asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(raw[v].x), "=r"(raw[v].y), "=r"(raw[v].z), "=r"(raw[v].w)
                         : "l"(xr + i)
                         : "memory");
            const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
#pragma unroll
            for (int e = 0; e < 4; ++e) { const float2 f = __half22float2(h[e]); s += f.x + f.y; }
        }
    }
    const float mean = block_sum_rt(s, red) / (float)D;
    float q = 0.f;
#pragma unroll
    for (int v = 0; v < LV_MAXV; ++v) {
        if (threadIdx.x + v * RT < nv) {
            const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(h[e]);
                q += (f.x - mean) * (f.x - mean) + (f.y - mean) * (f.y - mean);
            }
        }
    }
    const float rstd = rsqrtf(block_sum_rt(q, red) / (float)D + 1e-5f);
#pragma unroll
    for (int v = 0; v < LV_MAXV; ++v) {
        const int i = threadIdx.x + v * RT;
        if (i < nv && AB_BC(8 * (i + 1) <= D)) {
            const __half2 *h = reinterpret_cast<const __half2*>(&raw[v]), *wh = reinterpret_cast<const __half2*>(&wv[v]), *bh = reinterpret_cast<const __half2*>(&bv[v]);
            uint4 o;
            __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(h[e]), wf = __half22float2(wh[e]), bf = __half22float2(bh[e]);
                oh[e] = __floats2half2_rn((f.x - mean) * rstd * wf.x + bf.x, (f.y - mean) * rstd * wf.y + bf.y);
            }
            reinterpret_cast<uint4*>(out + m * D)[i] = o;
        }
    }
}

// For row m = (b, t): prev = t ? xn[m-1] : x_prev[b];  out_c[m] = xn[m] + (prev - xn[m]) * mix_c.
// With T == 1 the same block also stores the new token-shift state (x_prev[b] = xn[m]).
__global__ void __launch_bounds__(RT) mix_rows_kernel(MixParams p) {
    const size_t m = blockIdx.x;
    const int b = (int)(m / p.T), t = (int)(m % p.T);
    const __half* cur = p.xn + m * p.D;
    const __half* prev = t ? cur - p.D : p.x_prev + (size_t)b * p.D;
    for (int i = threadIdx.x; i < p.D; i += RT) {
        const float c = __half2float(cur[i]);
        const float d = rh(__half2float(prev[i]) - c);
        for (int j = 0; j < p.n_mix; ++j)
            p.out[j][m * p.D + i] = __float2half_rn(c + rh(d * __half2float(p.mix[j][i])));
        if (p.T == 1) p.x_prev[(size_t)b * p.D + i] = cur[i];
    }
}

// T == 1: layer norm and token-shift lerps of one row in one pass; the row stays in registers (16-byte loads and
// stores), the normalised row becomes the new token-shift state. Same rounding points as ln_rows + mix_rows.
constexpr int LM_MAXV = 4;   // 16-byte chunks per thread: D <= 8 * RT * LM_MAXV
constexpr int LM_TABLE_MAXV = 2;   // ... for sequences whose rows come from an embedding table
__global__ void __launch_bounds__(RT) ln_mix_rows_kernel(const __half* __restrict__ x, const __half* __restrict__ w,
                                                         const __half* __restrict__ b, const __grid_constant__ MixParams p,
                                                         int use_pdl) {
    __shared__ float red[RT / 32];
    const size_t m = blockIdx.x;
    const int nv = p.D / 8;
    const uint4* xr = reinterpret_cast<const uint4*>(x + m * p.D);
    uint4 raw[LM_MAXV], prv[LM_MAXV], wv_[LM_MAXV], bv_[LM_MAXV];
    float s = 0.f;
    // everything that does not depend on the row statistics is requested up front (norm weights into registers, the
    // lerp vectors into L1), so that the two block reductions are the only waits after the first load. Under
    // programmatic stream serialisation the parameters are requested while the preceding kernel still runs, and the
    // next kernel (a product, which starts with its weight stream) may start at once.
    if (use_pdl) pdl_launch_dependents();
#pragma unroll
    for (int v = 0; v < LM_MAXV; ++v) {
        const int i = threadIdx.x + v * RT;
        if (i < nv) {
            wv_[v] = reinterpret_cast<const uint4*>(w)[i];
            bv_[v] = reinterpret_cast<const uint4*>(b)[i];
#pragma unroll
            for (int j = 0; j < 6; ++j)
                if (j < p.n_mix) asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const uint4*>(p.mix[j]) + i));
        }
    }
    if (use_pdl) pdl_wait();
    if (p.table) xr = reinterpret_cast<const uint4*>(p.table + token_row(p.ids[m], p.vocab) * p.D);
#pragma unroll
    for (int v = 0; v < LM_MAXV; ++v) {
        const int i = threadIdx.x + v * RT;
        if (i < nv) {
            // an ordinary (coherent) load that stays behind the wait above: the row was written by the preceding kernel
            asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(raw[v].x), "=r"(raw[v].y), "=r"(raw[v].z), "=r"(raw[v].w)
                         : "l"(xr + i)
                         : "memory");
            if (p.table && AB_BC(m < (size_t)p.B && 8 * (i + 1) <= p.D)) reinterpret_cast<uint4*>(p.x_copy + m * p.D)[i] = raw[v];
            prv[v] = reinterpret_cast<const uint4*>(p.x_prev + m * p.D)[i];
            const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
#pragma unroll
            for (int e = 0; e < 4; ++e) { const float2 f = __half22float2(h[e]); s += f.x + f.y; }
        }
    }
    const float mean = block_sum_rt(s, red) / (float)p.D;
    float q = 0.f;
#pragma unroll
    for (int v = 0; v < LM_MAXV; ++v) {
        if (threadIdx.x + v * RT < nv) {
            const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(h[e]);
                q += (f.x - mean) * (f.x - mean) + (f.y - mean) * (f.y - mean);
            }
        }
    }
    const float rstd = rsqrtf(block_sum_rt(q, red) / (float)p.D + 1e-5f);
#pragma unroll
    for (int v = 0; v < LM_MAXV; ++v) {
        const int i = threadIdx.x + v * RT;
        if (i < nv) {
            const uint4 wv = wv_[v], bv = bv_[v];
            const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
            const __half2* wh = reinterpret_cast<const __half2*>(&wv);
            const __half2* bh = reinterpret_cast<const __half2*>(&bv);
            const __half2* ph = reinterpret_cast<const __half2*>(&prv[v]);
            uint4 xn;
            __half2* xh = reinterpret_cast<__half2*>(&xn);
            float c[8], d[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(h[e]), wf = __half22float2(wh[e]), bf = __half22float2(bh[e]);
                xh[e] = __floats2half2_rn((f.x - mean) * rstd * wf.x + bf.x, (f.y - mean) * rstd * wf.y + bf.y);
                const float2 cf = __half22float2(xh[e]), pf = __half22float2(ph[e]);
                c[2 * e] = cf.x; c[2 * e + 1] = cf.y;
                d[2 * e] = rh(pf.x - cf.x); d[2 * e + 1] = rh(pf.y - cf.y);
            }
            reinterpret_cast<uint4*>(p.x_prev + m * p.D)[i] = xn;
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                if (j < p.n_mix) {
                    const uint4 mv = reinterpret_cast<const uint4*>(p.mix[j])[i];
                    const __half2* mh = reinterpret_cast<const __half2*>(&mv);
                    uint4 o;
                    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 mf = __half22float2(mh[e]);
                        oh[e] = __floats2half2_rn(c[2 * e] + rh(d[2 * e] * mf.x), c[2 * e + 1] + rh(d[2 * e + 1] * mf.y));
                    }
                    reinterpret_cast<uint4*>(p.out[j] + m * p.D)[i] = o;
                }
            }
        }
    }
}

// T > 1: layer norm and token-shift lerps of sequences in one pass. A block takes p.R consecutive rows of one sequence: the
// normalised row of step t - 1 stays in registers as the shift of step t, only the row in front of the block's first is
// normalised twice. The block with a sequence's first rows is the only one that touches its token-shift state: it
// reads it for step 0 and stores the sequence's last normalised row at the end.
// What bounds it: 2 bytes in and 2 * n_mix out per element (768 rows x 4096, six lerps: 44 MB, about 7 us at the copy
// bandwidth), then the two block-wide sums per row. Alone on a cold cache 21 us there, 13.5 us with one lerp; the three
// passes it replaces (norm, lerps with 2-byte accesses, state hand-over) took 62 and 27 us.
// Rows of an embedding table are read here up to LM_TABLE_MAXV chunks; four per thread leave no registers for it (552 bytes of
// spills, none without), and rows that long are gathered by a pass of their own.
template <int V>   // 16-byte chunks per thread: D <= 8 * RT * V
__global__ void __launch_bounds__(RT) ln_mix_seq_kernel(const __half* __restrict__ x, const __half* __restrict__ w,
                                                        const __half* __restrict__ b, const __grid_constant__ MixParams p, int R,
                                                        int use_pdl) {
    __shared__ float red[RT / 32];
    const int n_chunks = (p.T + R - 1) / R, seq = blockIdx.x / n_chunks, t0 = (blockIdx.x - seq * n_chunks) * R;
    constexpr bool TABLE = V <= LM_TABLE_MAXV;
    const int nv = p.D / 8;
    const uint4* xs = reinterpret_cast<const uint4*>(x + (size_t)seq * p.T * p.D);
    uint4* state = reinterpret_cast<uint4*>(p.x_prev + (size_t)seq * p.D);
    if (use_pdl) pdl_launch_dependents();
    uint4 wv_[V], bv_[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int i = threadIdx.x + v * RT;
        if (i < nv) {
            wv_[v] = reinterpret_cast<const uint4*>(w)[i];
            bv_[v] = reinterpret_cast<const uint4*>(b)[i];
        }
    }
    if (use_pdl) pdl_wait();
    auto load = [&](int t, uint4* raw) {
        const uint4* row = xs + (size_t)t * nv;
        if (TABLE && p.table) row = reinterpret_cast<const uint4*>(p.table + token_row(p.ids[(size_t)seq * p.T + t], p.vocab) * p.D);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int i = threadIdx.x + v * RT;
            // an ordinary (coherent) load that stays behind the wait above: the row was written by the preceding kernel
            if (i < nv && AB_BC(seq < p.B && t >= 0 && t < p.T && 8 * (i + 1) <= p.D))
                asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(raw[v].x), "=r"(raw[v].y), "=r"(raw[v].z), "=r"(raw[v].w)
                             : "l"(row + i)
                             : "memory");
        }
    };
    auto norm = [&](const uint4* raw, uint4* xn) {   // same rounding points as ln_rows
        float s = 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            if (threadIdx.x + v * RT < nv) {
                const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
#pragma unroll
                for (int e = 0; e < 4; ++e) { const float2 f = __half22float2(h[e]); s += f.x + f.y; }
            }
        }
        const float mean = block_sum_rt(s, red) / (float)p.D;
        float q = 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            if (threadIdx.x + v * RT < nv) {
                const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __half22float2(h[e]);
                    q += (f.x - mean) * (f.x - mean) + (f.y - mean) * (f.y - mean);
                }
            }
        }
        const float rstd = rsqrtf(block_sum_rt(q, red) / (float)p.D + 1e-5f);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
            const __half2* wh = reinterpret_cast<const __half2*>(&wv_[v]);
            const __half2* bh = reinterpret_cast<const __half2*>(&bv_[v]);
            __half2* xh = reinterpret_cast<__half2*>(&xn[v]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(h[e]), wf = __half22float2(wh[e]), bf = __half22float2(bh[e]);
                xh[e] = __floats2half2_rn((f.x - mean) * rstd * wf.x + bf.x, (f.y - mean) * rstd * wf.y + bf.y);
            }
        }
    };
    const int t1 = min(t0 + R, p.T);
    uint4 raw[V], prev[V];
    if (t0 > 0) {
        load(t0 - 1, raw);
        norm(raw, prev);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (threadIdx.x + v * RT < nv && AB_BC(seq < p.B)) prev[v] = state[threadIdx.x + v * RT];
    }
    load(t0, raw);
    for (int t = t0; t < t1; ++t) {
        uint4 xn[V];
        norm(raw, xn);
        if (TABLE && p.table) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int i = threadIdx.x + v * RT;
                if (i < nv && AB_BC(seq < p.B && t < p.T && 8 * (i + 1) <= p.D))
                    reinterpret_cast<uint4*>(p.x_copy + ((size_t)seq * p.T + t) * p.D)[i] = raw[v];
            }
        }
        if (t + 1 < t1) load(t + 1, raw);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int i = threadIdx.x + v * RT;
            if (i < nv) {
                const __half2* ch = reinterpret_cast<const __half2*>(&xn[v]);
                const __half2* ph = reinterpret_cast<const __half2*>(&prev[v]);
                float c[8], d[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 cf = __half22float2(ch[e]), pf = __half22float2(ph[e]);
                    c[2 * e] = cf.x; c[2 * e + 1] = cf.y;
                    d[2 * e] = rh(pf.x - cf.x); d[2 * e + 1] = rh(pf.y - cf.y);
                }
                for (int j = 0; j < p.n_mix; ++j) {
                    const uint4 mv = reinterpret_cast<const uint4*>(p.mix[j])[i];
                    const __half2* mh = reinterpret_cast<const __half2*>(&mv);
                    uint4 o;
                    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 mf = __half22float2(mh[e]);
                        oh[e] = __floats2half2_rn(c[2 * e] + rh(d[2 * e] * mf.x), c[2 * e + 1] + rh(d[2 * e + 1] * mf.y));
                    }
                    if (AB_BC(seq < p.B && t >= t0 && t < p.T && j < 6 && 8 * (i + 1) <= p.D))
                        reinterpret_cast<uint4*>(p.out[j] + ((size_t)seq * p.T + t) * p.D)[i] = o;
                }
                prev[v] = xn[v];
            }
        }
    }
    if (t0 == 0) {   // the state read above is replaced by the normalised last row
        if (t1 < p.T) {
            load(p.T - 1, raw);
            norm(raw, prev);
        }
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (threadIdx.x + v * RT < nv && AB_BC(seq < p.B && 8 * (int)(threadIdx.x + v * RT + 1) <= p.D)) state[threadIdx.x + v * RT] = prev[v];
    }
}

// Greedy / noisy-greedy sampling of one token per row: argmax over the row of logit + U(0, noise)
// (reference/utils.py:43-45 adds uniform noise and takes the first entry of a descending argsort). Ties go to the
// lowest index. The noise is a counter-based hash of (seed, row, column): reproducible, not torch's generator.
__device__ __forceinline__ float sample_noise(uint32_t seed, uint32_t row, uint32_t col) {
    uint32_t x = seed ^ (row * 0x9E3779B9u) ^ (col * 0x85EBCA6Bu);
    x ^= x >> 16; x *= 0x7FEB352Du; x ^= x >> 15; x *= 0x846CA68Bu; x ^= x >> 16;
    return (float)(x >> 8) * (1.0f / 16777216.0f);   // [0, 1)
}
// What bounds it: reading the logits. The noise hash takes some fifteen integer operations, too many to draw it for every
// logit (320 rows of 65536: 28.8 us); so the row is read in batches of SR_U 16-byte chunks per thread, the batch's plain
// maximum over the block is taken first, and only chunks that can still reach it are looked at value by value: noise is
// never negative and always below `noise`, so a logit v ends up in [v, v + noise]. Skipped are chunks strictly below; ties
// and NaNs take the long way, the result is the same id.
// (With the maximum over a warp instead of the block, eight chunks per warp and batch still took the long way: 18.1 us, then 13.3.)
// NT threads per row: 1024 for up to 16 rows, whose rows are a batch of eight chunks per thread (8 rows of 65536: 4.5 us); more
// threads than that do not share an SM, so further rows take 512 threads as long as every row has an SM to itself and 256
// beyond, in batches of four chunks of which the next travels while one is looked at (in a graph 100 rows of 65536 8.6 -> 5.8 us,
// 200 of 50277 9.4 -> 7.8, 320 of 65536 11.0 -> 10.1; in calls one after the other, whose launches outweigh it, 12.4 -> 12.1).
template <class OutT, int NT>
__global__ void __launch_bounds__(NT) sample_rows_kernel(const __half* __restrict__ logits, int V, float noise, uint32_t seed,
                                                         OutT* __restrict__ out) {
    constexpr bool AHEAD = NT < 1024;
    constexpr int SR_U = AHEAD ? 4 : 8;
    __shared__ float bv[NT / 32], tops[2][NT / 32];
    __shared__ int bi[NT / 32];
    const size_t row = blockIdx.x;
    const __half* lr = logits + row * V;
    float best = -INFINITY, floor_ = -INFINITY;   // floor_: the row's result is at least this
    int idx = 0x7fffffff;
    auto take = [&](float v, int i) {
        if (noise > 0.f) v += noise * sample_noise(seed, (uint32_t)row, (uint32_t)i);
        if (v > best || (v == best && i < idx)) { best = v; idx = i; }
    };
    // elements up to the first 16-byte boundary, chunks of eight, the rest
    const int head = min(V, (int)((16 - ((uintptr_t)lr & 15)) & 15) / 2), nv = (V - head) / 8;
    if ((int)threadIdx.x < head && AB_BC((int)threadIdx.x < V)) take(__half2float(lr[threadIdx.x]), threadIdx.x);
    const uint4* body = reinterpret_cast<const uint4*>(lr + head);
    int buf = 0;
    uint4 nxt[SR_U];
    auto request = [&](int c0) {
#pragma unroll
        for (int u = 0; u < SR_U; ++u) {
            const int c = c0 + u * NT + threadIdx.x;
            if (c < nv && AB_BC(c >= 0 && head + 8 * (c + 1) <= V)) nxt[u] = __ldcs(body + c);
        }
    };
    if (AHEAD) request(0);
    for (int c0 = 0; c0 < nv; c0 += NT * SR_U, buf ^= 1) {   // uniform in the block
        uint4 q[SR_U];
        __half m[SR_U];
        if (!AHEAD) request(c0);
#pragma unroll
        for (int u = 0; u < SR_U; ++u) q[u] = nxt[u];
        if (AHEAD) request(c0 + NT * SR_U);   // the next batch travels while this one is looked at
        __half top = __ushort_as_half((unsigned short)0xfc00u);   // -inf
#pragma unroll
        for (int u = 0; u < SR_U; ++u) {
            m[u] = __ushort_as_half((unsigned short)0xfc00u);
            if (c0 + u * NT + (int)threadIdx.x < nv) {
                const __half2* h = reinterpret_cast<const __half2*>(&q[u]);
                const __half2 t = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
                m[u] = __hmax(__low2half(t), __high2half(t));
            }
            top = __hmax(top, m[u]);
        }
        const float wtop = warp_max(fmaxf(__half2float(top), best));
        if ((threadIdx.x & 31) == 0) tops[buf][threadIdx.x >> 5] = wtop;
        __syncthreads();   // the two buffers alternate: one barrier per batch
#pragma unroll
        for (int i = 0; i < NT / 32; ++i) floor_ = fmaxf(floor_, tops[buf][i]);
#pragma unroll
        for (int u = 0; u < SR_U; ++u) {
            const int c = c0 + u * NT + threadIdx.x;
            if (c < nv && !(__half2float(m[u]) + noise < floor_)) {
                const __half2* h = reinterpret_cast<const __half2*>(&q[u]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __half22float2(h[e]);
                    take(f.x, head + c * 8 + 2 * e);
                    take(f.y, head + c * 8 + 2 * e + 1);
                }
            }
        }
    }
    for (int i = head + nv * 8 + threadIdx.x; i < V; i += NT)
        if (AB_BC(i >= 0)) take(__half2float(lr[i]), i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
    }
    if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < NT / 32; ++w)
            if (bv[w] > best || (bv[w] == best && bi[w] < idx)) { best = bv[w]; idx = bi[w]; }
        out[row] = (OutT)idx;
    }
}

// x_prev[b] = xn[b, T-1]
__global__ void __launch_bounds__(RT) last_rows_kernel(const __half* __restrict__ xn, int T, int D, __half* __restrict__ x_prev) {
    const size_t b = blockIdx.x;
    for (int i = threadIdx.x; i < D; i += RT) x_prev[b * D + i] = xn[(b * T + T - 1) * D + i];
}

}  // namespace

int gather_rows(const __half* table, const int* idx, int rows, int D, int vocab, __half* out, cudaStream_t s) {
    AB_CHECK_ARG(table && idx && out && rows > 0 && D % 8 == 0 && vocab > 0, "gather_rows: bad argument");
    gather_rows_kernel<<<rows, RT, 0, s>>>(table, idx, D, vocab, out);
    AB_CUDA(cudaGetLastError());
    return OK;
}
int ln_rows(const __half* x, const __half* w, const __half* b, int rows, int D, int stride, int offset, __half* out,
            cudaStream_t s, bool pdl) {
    AB_CHECK_ARG(x && w && b && out && rows > 0, "ln_rows: bad argument");
    if (D % 8 == 0 && D <= 8 * RT * LV_MAXV && (((uintptr_t)x | (uintptr_t)w | (uintptr_t)b | (uintptr_t)out) & 15) == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(rows);
        cfg.blockDim = dim3(RT);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = pdl ? 1 : 0;
        AB_CUDA(cudaLaunchKernelEx(&cfg, ln_vec_kernel, x, w, b, D, stride, offset, out, pdl ? 1 : 0));
        return OK;
    }
    ln_rows_kernel<<<rows, RT, 0, s>>>(x, w, b, D, stride, offset, out);
    AB_CUDA(cudaGetLastError());
    return OK;
}
bool ln_mix_rows_ok(const __half* w, const __half* b, const MixParams& p) {
    uintptr_t any = (uintptr_t)w | (uintptr_t)b | (uintptr_t)p.x_prev;
    for (int j = 0; j < p.n_mix; ++j) any |= (uintptr_t)p.mix[j];
    return p.D % 8 == 0 && p.D <= 8 * RT * LM_MAXV && (any & 15) == 0;
}
bool ln_mix_table_ok(const __half* table, const MixParams& p) {
    return ((uintptr_t)table & 15) == 0 && (p.T == 1 || p.D <= 8 * RT * LM_TABLE_MAXV);
}
int ln_mix_rows(const __half* x, const __half* w, const __half* b, const MixParams& p, cudaStream_t s, bool pdl) {
    AB_CHECK_ARG(x && w && b && p.x_prev && p.n_mix >= 1 && p.n_mix <= 6 && p.B > 0 && ln_mix_rows_ok(w, b, p), "ln_mix_rows: bad argument");
    AB_CHECK_ARG(!p.table || (p.ids && p.x_copy && p.vocab > 0 && ln_mix_table_ok(p.table, p)), "ln_mix_rows: bad embedding table");
    // rows per block of a sequence: as few as fill the GPU (each block normalises one row more than it owns)
    const int rows = p.B * p.T, R = rows >= 2048 ? 4 : (rows >= 512 ? 2 : 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.T == 1 ? p.B : p.B * ((p.T + R - 1) / R));
    cfg.blockDim = dim3(RT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    if (p.T == 1) AB_CUDA(cudaLaunchKernelEx(&cfg, ln_mix_rows_kernel, x, w, b, p, pdl ? 1 : 0));
    else if (p.D <= 8 * RT * 2) AB_CUDA(cudaLaunchKernelEx(&cfg, ln_mix_seq_kernel<2>, x, w, b, p, R, pdl ? 1 : 0));
    else AB_CUDA(cudaLaunchKernelEx(&cfg, ln_mix_seq_kernel<LM_MAXV>, x, w, b, p, R, pdl ? 1 : 0));
    return OK;
}
int sample_rows(const __half* logits, int rows, int V, float noise, uint32_t seed, void* out, bool out_i64, cudaStream_t s) {
    AB_CHECK_ARG(logits && out && rows > 0 && V > 0 && noise >= 0.f, "sample_rows: bad argument");
    if (rows <= 16) {
        if (out_i64) sample_rows_kernel<long long, 1024><<<rows, 1024, 0, s>>>(logits, V, noise, seed, (long long*)out);
        else sample_rows_kernel<int, 1024><<<rows, 1024, 0, s>>>(logits, V, noise, seed, (int*)out);
    } else if (rows <= current_sm_count()) {
        if (out_i64) sample_rows_kernel<long long, 512><<<rows, 512, 0, s>>>(logits, V, noise, seed, (long long*)out);
        else sample_rows_kernel<int, 512><<<rows, 512, 0, s>>>(logits, V, noise, seed, (int*)out);
    } else {
        if (out_i64) sample_rows_kernel<long long, 256><<<rows, 256, 0, s>>>(logits, V, noise, seed, (long long*)out);
        else sample_rows_kernel<int, 256><<<rows, 256, 0, s>>>(logits, V, noise, seed, (int*)out);
    }
    AB_CUDA(cudaGetLastError());
    return OK;
}
int mix_rows(const MixParams& p, cudaStream_t s) {
    AB_CHECK_ARG(p.xn && p.x_prev && p.n_mix >= 1 && p.n_mix <= 6 && p.B > 0 && p.T > 0, "mix_rows: bad argument");
    mix_rows_kernel<<<p.B * p.T, RT, 0, s>>>(p);
    AB_CUDA(cudaGetLastError());
    if (p.T > 1) {
        last_rows_kernel<<<p.B, RT, 0, s>>>(p.xn, p.T, p.D, p.x_prev);
        AB_CUDA(cudaGetLastError());
    }
    return OK;
}

}  // namespace ab

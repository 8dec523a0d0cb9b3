// Batched products of few rows (up to 24): weights streamed past resident activations, mma.sync.
//
//   Y[rows, n_out] = X[rows, k] W^T       (the products of gemm.cu, same formats, roundings and epilogues)
//
// What bounds it: reading the weights. A tile of gemm.cu keeps a block busy for its launch, its pipeline's fill, a hand-over
// between warps of 390 cycles a k-step and the exchange of a split K, none of which a few rows of activations hide. Here the
// activations of a block's share of K lie in shared memory (TMA, 128-byte swizzle) for its whole life, and its warps stream
// tiles of 32 weight rows past them, each with a ring of its own: its first lane asks for 4 KB pieces (32 rows x 128 bytes), four
// ahead, which is 128 KB per SM; nobody else is waited for until a tile is done. The first pieces are requested before the
// wait for the preceding grid. `kw` warps share a tile's K (8 / kw tiles are under way at a time); where the activations do not fit,
// a cluster of `ks` blocks splits K. A lane's 16 bytes of a row are its own inner indices of several MMAs (16 rows x 8 batch
// rows x 16), in the order in which they lie in memory, and the activations are read in the same order: nothing is moved
// between lanes. Partial sums meet in shared memory, those of a cluster through distributed shared memory, in one order always.
// In the step of 8 sequences (int8, 4096 wide) the r/k/v launch moves its 58 MB in 11 us of its 13, the ffn key its 67 in 11.3 of 16;
// the whole step of two blocks 243 -> 177 us. (Weights straight into registers, 8 KB a warp in flight: 203. 16 warps with two pieces
// each: 175, and up to 1.5 us slower alone on small matrices. Tiles of 16 rows, which divide better: 195 - 203, they read the
// activations twice as often. The code of a launch is fetched cold: a tile's end unrolled four times cost 0.7 us a launch.)
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "gemm.cuh"
#include "gemv.cuh"

namespace ab {

namespace {

constexpr int SG_WARPS = 8, SG_THREADS = 32 * SG_WARPS;
constexpr int SG_ROWS = 32;             // weight rows of a tile: two MMAs share what is read of the activations
constexpr int SG_PIECE = SG_ROWS * 128, SG_PIECE_SC = SG_ROWS * 16;   // a stage of a warp's ring: 128 bytes of each row, NVFP4 scales
constexpr int SG_COL = SG_ROWS + 4;     // a column of partial sums with padding: written and read without bank conflicts
constexpr int SG_STAGES = 4;            // at most
constexpr int SG_MAX_ROWS = 24;
constexpr int SG_SMEM = 225 * 1024;

struct SgProb {
    const void* scale;
    const __half* resid;
    __half* y;
    float tscale;
    int fmt, epi, n_out, k, n_tiles, kw, sc_map;
};
struct SgGroup {
    int cl_base[8];        // first cluster of each product, and the end
    SgProb pr[7];
    int n, rows, ks, stages, stage_bytes;
    int x_bytes, ring_bytes, red_bytes;   // shared memory: activations, rings, partial sums of the warps (and, ks > 1, of the block's tiles)
};
struct SgMaps {
    CUtensorMap x[7], w[7], s[7];
};
static_assert(sizeof(SgMaps) + sizeof(SgGroup) <= 4096, "parameters of the stream kernel");

// K is dealt out in pieces: 128 bytes of a row, which are two, four or one tiles of 64 activations
__host__ __device__ constexpr int sg_tiles(int fmt) { return fmt == FMT_I8 ? 2 : fmt == FMT_FP4 ? 4 : 1; }
__host__ __device__ constexpr int sg_pieces(int fmt, int k) { return (k + 64 * sg_tiles(fmt) - 1) / (64 * sg_tiles(fmt)); }

__device__ __forceinline__ void mma_f16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// int8 -> fp16 exactly (see raw_dequant)
__device__ __forceinline__ void i8x4_to_half2x2(uint32_t w, uint32_t* h) {
    const uint32_t x = w ^ 0x80808080u;
    const uint32_t lo = __byte_perm(x, 0x64646464u, 0x4140), hi = __byte_perm(x, 0x64646464u, 0x4342);
    const __half2 bias = __floats2half2_rn(1152.f, 1152.f);
    const __half2 l = __hsub2(*reinterpret_cast<const __half2*>(&lo), bias), u = __hsub2(*reinterpret_cast<const __half2*>(&hi), bias);
    h[0] = *reinterpret_cast<const uint32_t*>(&l);
    h[1] = *reinterpret_cast<const uint32_t*>(&u);
}
__device__ __forceinline__ void fp4x8_to_half2x4(uint32_t w, __half2 s, uint32_t* h) {
    e2m1x8_to_half2x4(w, h);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const __half2 v = __hmul2(*reinterpret_cast<const __half2*>(&h[e]), s);   // exact in fp16
        h[e] = *reinterpret_cast<const uint32_t*>(&v);
    }
}
__device__ __forceinline__ float sg_peer_ld(const float* own, uint32_t rank) {
    float v;
    asm volatile("{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %1, %2;\n ld.shared::cluster.f32 %0, [a];\n}" : "=f"(v) : "r"(smem_u32(own)), "r"(rank) : "memory");
    return v;
}

__device__ __forceinline__ void sg_tma(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

// NT: batch rows in eights
template <int NT>
__global__ void __launch_bounds__(SG_THREADS, 1) stream_kernel(const __grid_constant__ SgMaps maps, const __grid_constant__ SgGroup g) {
    extern __shared__ __align__(1024) unsigned char ssm[];
    __shared__ uint64_t x_full[SG_WARPS], w_full[SG_WARPS][SG_STAGES];
    __shared__ uint32_t s_nobody;
    constexpr int N = 8 * NT, TILE_F = N * SG_COL;   // floats of a tile's partial sums: [batch row][weight row]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q = lane & 3;
    const int cl = (int)blockIdx.x / g.ks, rank = (int)blockIdx.x - cl * g.ks;
    int pi = 0;
    while (pi + 1 < g.n && cl >= g.cl_base[pi + 1]) ++pi;
    const SgProb& pb = g.pr[pi];
    const int n_cl = g.cl_base[pi + 1] - g.cl_base[pi], local = cl - g.cl_base[pi];
    const int t0 = (int)((long long)pb.n_tiles * local / n_cl), t1 = (int)((long long)pb.n_tiles * (local + 1) / n_cl);
    const int fmt = pb.fmt, n_pieces = sg_pieces(fmt, pb.k), xt = sg_tiles(fmt);
    const int p0 = n_pieces * rank / g.ks, np = n_pieces * (rank + 1) / g.ks - p0;          // this block's pieces of K
    const int kw = pb.kw, slot = warp / kw, kwi = warp - slot * kw, tpr = SG_WARPS / kw;
    const int c0 = np * kwi / kw, nc = np * (kwi + 1) / kw - c0;                            // this warp's, counted from p0
    const int rounds = t0 + slot < t1 ? (t1 - t0 - slot + tpr - 1) / tpr : 0, total = rounds * nc;
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)ssm + 1023) & ~(uintptr_t)1023);
    unsigned char* sx = base;                                                  // activation tiles from piece p0 on: N rows x 128 bytes
    unsigned char* ring = base + g.x_bytes + warp * g.stages * SG_PIECE;       // this warp's stages, and their scales behind all rings
    unsigned char* ring_sc = base + g.x_bytes + SG_WARPS * g.stages * SG_PIECE + warp * g.stages * SG_PIECE_SC;
    float* red = reinterpret_cast<float*>(base + g.x_bytes + g.ring_bytes);
    float* bpart = reinterpret_cast<float*>(base + g.x_bytes + g.ring_bytes + g.red_bytes);
    if (lane == 0) {
        mbar_init(&x_full[warp], 1);
        for (int s = 0; s < g.stages; ++s) mbar_init(&w_full[warp][s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_launch_dependents();
    // The warp's pieces one behind the other, tile after tile; its first lane requests them, g.stages ahead of the one worked on.
    int in_i = 0, in_c = 0, in_row = (t0 + slot) * SG_ROWS, in_stage = 0;
    auto request = [&]() {   // (one lane)
        if (in_i >= total) return;
        uint64_t* bar = &w_full[warp][in_stage];
        mbar_expect_tx(bar, (uint32_t)(SG_PIECE + (pb.sc_map ? SG_PIECE_SC : 0)));
        sg_tma(ring + in_stage * SG_PIECE, &maps.w[pi], (p0 + c0 + in_c) * 128, in_row, bar);
        if (pb.sc_map) sg_tma(ring_sc + in_stage * SG_PIECE_SC, &maps.s[pi], (p0 + c0 + in_c) * 16, in_row, bar);
        ++in_i;
        if (++in_stage == g.stages) in_stage = 0;
        if (++in_c == nc) { in_c = 0; in_row += tpr * SG_ROWS; }
    };
    if (lane == 0)   // weights are never written: they travel while the preceding grid still runs
        for (int s = 0; s < g.stages; ++s) request();
    pdl_wait();
    if (slot == 0 && lane == 0) {   // activations: the warps of the first tile slot fetch their own share (a tile beyond K arrives as zeros)
        mbar_expect_tx(&x_full[kwi], (uint32_t)(nc * xt * N * 128));
        for (int t = c0 * xt; t < (c0 + nc) * xt; ++t) sg_tma(sx + t * (N * 128), &maps.x[pi], (p0 * xt + t) * 64, 0, &x_full[kwi]);
    }
    __syncwarp();
    bool failed = !mbar_wait_bounded(&x_full[kwi], 0u, 1u << 16);

    auto run = [&](auto fmt_c) {
        constexpr int F = decltype(fmt_c)::value, XT = sg_tiles(F);
        float acc[2][NT][4];
        auto clear = [&]() {
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int n = 0; n < NT; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;
        };
        // Two steps of 16 inner indices: eight weights of rows gq and gq + 8 of both halves of the tile (l, h) against the same
        // inputs of batch row gq: 16-byte piece `piece` of activation tile kt.
        auto step = [&](const uint32_t (*l)[4], const uint32_t (*h)[4], int kt, int piece) {
            if (!AB_BC(kt >= 0 && (kt + 1) * N * 128 <= g.x_bytes && piece >= 0 && piece < 8)) return;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const uint4 x = *reinterpret_cast<const uint4*>(sx + kt * (N * 128) + (n * 8 + gq) * 128 + ((piece ^ gq) << 4));
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    mma_f16(acc[m][n], l[m][0], h[m][0], l[m][1], h[m][1], x.x, x.y);
                    mma_f16(acc[m][n], l[m][2], h[m][2], l[m][3], h[m][3], x.z, x.w);
                }
            }
        };
        // (returns a combination of a word of each load from the stage)
        auto piece = [&](const unsigned char* w, const unsigned char* sc, int c, int row0) -> uint32_t {
            (void)sc; (void)row0;
            uint32_t used = 0;
#pragma unroll
            for (int i = 0; i < 2; ++i) {   // halves of the 128 bytes: a lane's 16 bytes of four rows
                uint4 lo[2], hi[2];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    lo[m] = *reinterpret_cast<const uint4*>(w + (16 * m + gq) * 128 + (((4 * i + q) ^ gq) << 4));
                    hi[m] = *reinterpret_cast<const uint4*>(w + (16 * m + 8 + gq) * 128 + (((4 * i + q) ^ gq) << 4));
                    used ^= lo[m].x ^ hi[m].x;
                }
                uint32_t l[2][4], h[2][4];
                if (F == FMT_I8) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            i8x4_to_half2x2(j ? lo[m].z : lo[m].x, l[m]); i8x4_to_half2x2(j ? lo[m].w : lo[m].y, l[m] + 2);
                            i8x4_to_half2x2(j ? hi[m].z : hi[m].x, h[m]); i8x4_to_half2x2(j ? hi[m].w : hi[m].y, h[m] + 2);
                        }
                        step(l, h, c * XT + i, 2 * q + j);
                    }
                } else if (F == FMT_F16) {
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        l[m][0] = lo[m].x; l[m][1] = lo[m].y; l[m][2] = lo[m].z; l[m][3] = lo[m].w;
                        h[m][0] = hi[m].x; h[m][1] = hi[m].y; h[m][2] = hi[m].z; h[m][3] = hi[m].w;
                    }
                    step(l, h, c, 4 * i + q);
                } else {
                    __half2 sl[2], sh[2];   // the two block scales of a lane's 32 inputs
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        uint32_t a, b;
                        if (sc) {
                            a = *reinterpret_cast<const unsigned short*>(sc + (16 * m + gq) * 16 + i * 8 + 2 * q);
                            b = *reinterpret_cast<const unsigned short*>(sc + (16 * m + 8 + gq) * 16 + i * 8 + 2 * q);
                        } else {   // no map for them (k not a multiple of 256)
                            const int at = (p0 + c) * 16 + i * 8 + 2 * q, pitch = pb.k / 16;
                            const unsigned char* s = reinterpret_cast<const unsigned char*>(pb.scale);
                            const int ra = row0 + 16 * m + gq, rb = ra + 8;
                            a = at < pitch && ra < pb.n_out ? __ldg(reinterpret_cast<const unsigned short*>(s + (size_t)ra * pitch + at)) : 0u;
                            b = at < pitch && rb < pb.n_out ? __ldg(reinterpret_cast<const unsigned short*>(s + (size_t)rb * pitch + at)) : 0u;
                        }
                        used ^= a ^ b;
                        sl[m] = e4m3x2_to_half2(a);
                        sh[m] = e4m3x2_to_half2(b);
                    }
                    // four words of eight inputs; lanes of the second activation tile (q >= 2) take them in the order 2, 3, 0, 1,
                    // so that the eight lanes of a shared-memory access find eight different bank groups
                    const bool swap = q >= 2;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool second = (j >= 2) != swap;   // which of the two scale blocks
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            const uint32_t wl[4] = {lo[m].x, lo[m].y, lo[m].z, lo[m].w}, wh[4] = {hi[m].x, hi[m].y, hi[m].z, hi[m].w};
                            fp4x8_to_half2x4(swap ? wl[j ^ 2] : wl[j], second ? __high2half2(sl[m]) : __low2half2(sl[m]), l[m]);
                            fp4x8_to_half2x4(swap ? wh[j ^ 2] : wh[j], second ? __high2half2(sh[m]) : __low2half2(sh[m]), h[m]);
                        }
                        step(l, h, c * XT + 2 * i + (q >> 1), (q & 1) * 4 + (swap ? j ^ 2 : j));
                    }
                }
            }
            return used;
        };
        // A lane finishes one weight row for some of the batch rows: 64 consecutive bytes a warp and batch row.
        auto scale_of = [&](int row) {
            if (F != FMT_I8) return pb.tscale;
            return row < pb.n_out ? __ldg(reinterpret_cast<const float*>(pb.scale) + row) : 0.f;
        };
        auto store = [&](int row, int n, float v, float scale, __half resid) {
            if (!(row < pb.n_out && n < g.rows) || !AB_BC(row >= 0 && n >= 0)) return;
            __half* y = pb.y + (size_t)n * pb.n_out + row;
            if (pb.epi == EPI_RESID) *y = __hadd(resid, __float2half_rn(v * scale));
            else *y = __float2half_rn(apply_epi(pb.epi, rh(v * scale)));
        };
        auto resid_of = [&](int row, int n) { return pb.epi == EPI_RESID && row < pb.n_out && n < g.rows ? pb.resid[(size_t)n * pb.n_out + row] : __half(0.f); };
        int stage = 0, i = 0;
        uint32_t parity = 0;
        clear();
        for (int round = 0; round < rounds; ++round) {
            const int tile = t0 + slot + round * tpr, row = tile * SG_ROWS + lane;
            const float scale = scale_of(row);   // (used at the end of the tile)
            for (int c = 0; c < nc; ++c, ++i) {
                if (!failed && !mbar_wait_bounded(&w_full[warp][stage], parity, 1u << 16)) failed = true;
                const uint32_t used = piece(ring + stage * SG_PIECE, F == FMT_FP4 && pb.sc_map ? ring_sc + stage * SG_PIECE_SC : nullptr, c0 + c, tile * SG_ROWS);
                loads_returned(used, &s_nobody);
                __syncwarp();   // every lane has read the stage
                if (lane == 0 && !failed) request();
                if (++stage == g.stages) { stage = 0; parity ^= 1u; }
            }
            // the tile's sums: the warps that share it leave theirs in shared memory and add them in the order of K
            if (round > 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(kw * 32) : "memory");   // the tile before has been read
            float* mine = red + warp * TILE_F;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (AB_BC((warp + 1) * TILE_F * 4 <= g.red_bytes)) mine[(n * 8 + 2 * q + (e & 1)) * SG_COL + 16 * m + gq + 8 * (e >> 1)] = acc[m][n][e];
            clear();
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(kw * 32) : "memory");
            const float* first = red + slot * kw * TILE_F + lane;
#pragma unroll 1
            for (int n = kwi; n < N; n += kw) {
                float v = 0.f;
#pragma unroll 4
                for (int e = 0; e < kw; ++e) v += first[e * TILE_F + n * SG_COL];
                if (g.ks > 1) bpart[(tile - t0) * TILE_F + n * SG_COL + lane] = v;
                else store(row, n, v, scale, resid_of(row, n));
            }
        }
        if (g.ks > 1) {   // the blocks of a cluster finish its tiles in turn
            asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
            for (int t = rank; t < t1 - t0; t += g.ks) {
                const int row = (t0 + t) * SG_ROWS + lane;
                const float scale = scale_of(row);
#pragma unroll 1
                for (int n = warp; n < N; n += SG_WARPS) {
                    const __half resid = resid_of(row, n);
                    float v = 0.f;
                    for (int r = 0; r < g.ks; ++r) v += sg_peer_ld(bpart + t * TILE_F + n * SG_COL + lane, (uint32_t)r);
                    store(row, n, v, scale, resid);
                }
            }
            asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    };
    if (fmt == FMT_I8) run(std::integral_constant<int, FMT_I8>());
    else if (fmt == FMT_FP4) run(std::integral_constant<int, FMT_FP4>());
    else run(std::integral_constant<int, FMT_F16>());
    if (failed) {   // (copies on their way still find their shared memory)
        if (lane == 0) atomicOr(&g_device_status, DEV_WAIT_GEMM);
        for (int s = 0; s < 100; ++s) __nanosleep(1000);
    }
}

// How a launch is dealt out.
struct SgShape {
    int ks, n_cl[7], kw[7], x_bytes, ring_bytes, red_bytes, stages, smem;
};
// Where this kernel is the faster one, measured in graphs of launches over rotating matrices (this kernel and gemm.cu's, us):
//   up to 8 rows everywhere (int8 4096 x 4096 8.8 and 13.2, 16384 x 4096 17.9 and 19.3, 4096 x 16384 18.8 and 23.3, 65536 x 1024 20.7
//     and 28.8; nvfp4 6.8 and 11.8, 17.3 and 18.0, 18.4 and 22.6, 20.0 and 28.0; fp16 9.9 and 14.2), but for large fp16 matrices, whose
//     k-steps are long enough to hide the hand-over there (10240 x 2560 15.6 and 12.8);
//   up to 16 rows for matrices of 17 M weights (int8 2560 x 2560 6.9 and 10.1, 1024 x 16384 15.8 and 16.6, 4096 x 4096 12.4 and 13.2,
//     16384 x 4096 28 and 19; nvfp4 7.2 and 10.1, 12.5 and 15.5, 9.8 and 11.8; fp16 9.0 and 11.0);
//   up to 24 for small ones (2048 x 2048 int8 7.2 and 10.0, nvfp4 6.8 and 10.0, fp16 8.5 and 9.8; 1024 x 4096 7.7 and 10.8, 9.0 and 10.9, 8.3
//     and 10.8; 2560 x 2560 int8 12.0 and 11.3).
// In 16 shapes of 768 x 768 to 65536 x 1024, three formats, 2 to 24 rows, it is nowhere the slower one by more than 1 %. From 9 rows on
// the K split that the plan takes costs more than the planner's constants say (int8 4096 x 4096, 16 rows: 9.5 us in blocks that keep the
// whole of K, 12.2 and 16.7 in clusters of four and eight). Many tiles with little K (adapters) cost a round of sums each: 8.6 and 6
// in the step of a batch.
bool stream_pays(const GemmOp* ops, int n, int rows, int n_sm) {
    long long elems = 0, f16 = 0, tiles = 0, pieces = 0;
    for (int i = 0; i < n; ++i) {
        const long long t = (ops[i].w.n_out + SG_ROWS - 1) / SG_ROWS;
        elems += (long long)ops[i].w.n_out * ops[i].w.k;
        if (ops[i].w.fmt == FMT_F16) f16 += (long long)ops[i].w.n_out * ops[i].w.k;
        tiles += t;
        pieces += t * sg_pieces(ops[i].w.fmt, ops[i].w.k);
    }
    if (tiles > n_sm && pieces < 4 * tiles) return false;
    if (rows <= 8) return f16 <= 24000000;
    if (rows <= 16) return elems <= 17000000 && f16 <= 12000000;
    return rows <= SG_MAX_ROWS && elems <= 4500000 && elems >= 300000;
}
// clusters[log2(ks)]: clusters of ks blocks that fit the GPU at once. Times in cycles: a block moves a 4 KB piece in some 90 (the
// copy bandwidth over all SMs), its warps share that; the sums of a tile, the exchange of a cluster and the activations come on top.
bool stream_shape(const GemmOp* ops, int n, int rows, const int* clusters, SgShape* out) {
    if (n > 7 || !stream_pays(ops, n, rows, clusters[0])) return false;
    const int nt = (rows + 7) / 8, N = 8 * nt;
    bool any_fp4 = false;
    for (int i = 0; i < n; ++i) any_fp4 |= ops[i].w.fmt == FMT_FP4;
    long long best = 0;
    for (int lk = 0; lk < 4; ++lk) {
        const int ks = 1 << lk, total = clusters[lk];
        if (total < n) continue;
        SgShape s = {};
        s.ks = ks;
        s.red_bytes = SG_WARPS * SG_COL * N * 4;
        int pieces[7], tiles[7];   // of a block's share of a tile; tiles of a product
        for (int i = 0; i < n; ++i) {
            pieces[i] = (sg_pieces(ops[i].w.fmt, ops[i].w.k) + ks - 1) / ks;
            tiles[i] = (ops[i].w.n_out + SG_ROWS - 1) / SG_ROWS;
            s.n_cl[i] = 1;
            s.x_bytes = std::max(s.x_bytes, pieces[i] * sg_tiles(ops[i].w.fmt) * N * 128);
        }
        constexpr int PIECE = 90, TILE = 400;
        auto share = [&](int i, int tpc, int kw) {   // cycles of a block's `tpc` tiles, kw warps on each
            const int tpr = SG_WARPS / kw, rounds = (tpc + tpr - 1) / tpr;
            return (long long)rounds * (((pieces[i] + kw - 1) / kw) * (PIECE * SG_WARPS) + TILE + 12 * N);
        };
        int at[7] = {};   // the tiles of a block that `left` and `kw` stand for
        long long left[7];
        auto most = [&](int i) {
            const int tpc = (tiles[i] + s.n_cl[i] - 1) / s.n_cl[i];
            if (tpc == at[i]) return left[i];
            at[i] = tpc;
            long long b = 0;
            for (int kw = SG_WARPS; kw >= SG_WARPS / 8; kw /= 2) {
                const long long c = share(i, tpc, kw);
                if (b == 0 || c < b) { b = c; s.kw[i] = kw; }
            }
            return b;
        };
        // the clusters go where the largest share is left
        if (n == 1) s.n_cl[0] = std::min(tiles[0], total);
        for (int i = 0; i < n; ++i) left[i] = most(i);
        for (int used = n; n > 1 && used < total; ++used) {
            int pick = -1;
            for (int i = 0; i < n; ++i)
                if (s.n_cl[i] < tiles[i] && (pick < 0 || left[i] > left[pick])) pick = i;
            if (pick < 0) break;
            ++s.n_cl[pick];
            left[pick] = most(pick);
        }
        int bpart = 0;
        long long cost = 0;
        for (int i = 0; i < n; ++i) {
            if (ks > 1) bpart = std::max(bpart, (tiles[i] + s.n_cl[i] - 1) / s.n_cl[i] * SG_COL * N * 4);
            cost = std::max(cost, left[i]);
        }
        cost += s.x_bytes / 64 + (ks > 1 ? 2500 : 0);
        const int stage = SG_WARPS * (SG_PIECE + (any_fp4 ? SG_PIECE_SC : 0));
        const int room = SG_SMEM - 1024 - s.x_bytes - s.red_bytes - bpart;
        s.stages = std::min(SG_STAGES, room > 0 ? room / stage : 0);
        if (s.stages < 2) continue;
        const int in_flight = s.stages * SG_WARPS * SG_PIECE;
        if (in_flight < 128 * 1024) cost += cost * (128 * 1024 - in_flight) / (256 * 1024);
        s.ring_bytes = s.stages * stage;
        s.smem = s.x_bytes + s.ring_bytes + s.red_bytes + bpart + 1024;
        if (best == 0 || cost < best) { best = cost; *out = s; }
    }
    return best > 0;
}

typedef void (*SgKernel)(const SgMaps, const SgGroup);
SgKernel sg_kernel(int nt) { return nt == 1 ? stream_kernel<1> : nt == 2 ? stream_kernel<2> : stream_kernel<3>; }

}  // namespace

// Takes the launch if it has few enough rows; *taken says so. Arguments have been checked.
int stream_group_launch(const GemmOp* ops, int n, int rows, cudaStream_t stream, bool pdl, bool* taken) {
    *taken = false;
    if (rows > SG_MAX_ROWS) return OK;
    struct Clusters { int n[4]; };
    static std::mutex mu;
    static bool known[AB_MAX_DEVICES][4];
    static Clusters fit[AB_MAX_DEVICES][4];
    int dev = 0;
    AB_CUDA(cudaGetDevice(&dev));
    AB_CHECK_ARG(dev >= 0 && dev < AB_MAX_DEVICES, "gemm: device index %d not supported", dev);
    const int nt = (rows + 7) / 8;
    Clusters cf;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!known[dev][nt]) {
            AB_CUDA(cudaFuncSetAttribute(sg_kernel(nt), cudaFuncAttributeMaxDynamicSharedMemorySize, SG_SMEM));
            for (int lk = 0; lk < 4; ++lk) {
                cudaLaunchConfig_t c = {};
                c.gridDim = dim3(1 << lk);
                c.blockDim = dim3(SG_THREADS);
                c.dynamicSmemBytes = SG_SMEM;
                cudaLaunchAttribute a[1];
                a[0].id = cudaLaunchAttributeClusterDimension;
                a[0].val.clusterDim.x = 1 << lk;
                a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
                c.attrs = a;
                c.numAttrs = 1;
                AB_CUDA(cudaOccupancyMaxActiveClusters(&fit[dev][nt].n[lk], sg_kernel(nt), &c));
            }
            known[dev][nt] = true;
        }
        cf = fit[dev][nt];
    }
    SgShape sh;
    if (!stream_shape(ops, n, rows, cf.n, &sh)) return OK;
    EncodeTiledFn encode;
    const int st = get_encode_fn(&encode);
    if (st != OK) return st;
    SgMaps maps;
    SgGroup g = {};
    g.n = n; g.rows = rows; g.ks = sh.ks; g.stages = sh.stages;
    g.x_bytes = sh.x_bytes; g.ring_bytes = sh.ring_bytes; g.red_bytes = sh.red_bytes;
    int cl = 0;
    for (int i = 0; i < n; ++i) {
        const ab_mat& m = ops[i].w;
        SgProb& pb = g.pr[i];
        pb.scale = m.scale; pb.tscale = m.tscale;
        pb.resid = ops[i].resid; pb.y = ops[i].y; pb.epi = ops[i].epi;
        pb.fmt = m.fmt; pb.n_out = m.n_out; pb.k = m.k; pb.n_tiles = (m.n_out + SG_ROWS - 1) / SG_ROWS; pb.kw = sh.kw[i];
        g.cl_base[i] = cl;
        cl += sh.n_cl[i];
        auto map2d = [&](CUtensorMap* map, CUtensorMapDataType type, const void* p, cuuint64_t width, cuuint64_t height, cuuint64_t pitch,
                         cuuint32_t bw, cuuint32_t bh, bool swizzle) {
            const cuuint64_t dim[2] = {width, height}, stride[1] = {pitch};
            const cuuint32_t box[2] = {bw, bh}, estr[2] = {1, 1};
            const CUresult cr = encode(map, type, 2, const_cast<void*>(p), dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                       swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (cr == CUDA_SUCCESS) return (int)OK;
            set_error("gemm: cuTensorMapEncodeTiled failed with %d (rows=%d n_out=%d k=%d)", (int)cr, rows, m.n_out, m.k);
            return (int)ERR_CUDA;
        };
        const cuuint64_t row_bytes = m.fmt == FMT_F16 ? 2ull * m.k : m.fmt == FMT_I8 ? (cuuint64_t)m.k : m.k / 2;
        pb.sc_map = m.fmt == FMT_FP4 && m.k % 256 == 0 && ((uintptr_t)m.scale & 15) == 0 ? 1 : 0;
        int e = map2d(&maps.x[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, ops[i].x, m.k, rows, 2ull * m.k, 64, nt * 8, true);
        if (e == OK) e = map2d(&maps.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, m.w, row_bytes, m.n_out, row_bytes, 128, SG_ROWS, true);
        if (e == OK && pb.sc_map) e = map2d(&maps.s[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, m.scale, m.k / 16, m.n_out, m.k / 16, 16, SG_ROWS, false);
        if (e != OK) return e;
    }
    g.cl_base[n] = cl;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cl * sh.ks);
    cfg.blockDim = dim3(SG_THREADS);
    cfg.dynamicSmemBytes = sh.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (pdl) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (sh.ks > 1) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = sh.ks;
        attr[n_attr].val.clusterDim.y = attr[n_attr].val.clusterDim.z = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    AB_CUDA(cudaLaunchKernelEx(&cfg, sg_kernel(nt), maps, g));
    *taken = true;
    return OK;
}

}  // namespace ab

// Batched matrix products of the RWKV-7 batch path on the 5th-generation tensor cores (tcgen05 / TMEM),
// and the de-quantisation dump.
//
// Replaces the `[B,T,D] @ W` call sites of reference/rwkv7.py:283-288, :293, :300 (time-mix), :322-323
// (channel-mix) and :220 (vocabulary head) with weight-only int8 / NVFP4 / fp16 weights.
//
//   D[128 weight rows, N batch rows] (fp32, TMEM) += A[128, 64] (weights, fp16) * B[N, 64]^T (activations, fp16)
//
// The weights are the M side of the MMA so that every weight byte is read from HBM exactly once per
// N tile; the batch (up to 320 rows per block: an MMA of N = 192 and one for the rest) is the N side.
//   weight warp: brings raw quantised rows in with TMA, 128 bytes of each of the 128 rows at a time (2 k-steps of int8, 4 of
//               NVFP4 with their block scales beside them, 1 of fp16), into as many shared-memory slots as the activation
//               stages leave room for; no producer computes an address or waits for a copy of its own.
//   producer groups (G_NG groups of 4 warps; thread = one of the block's 128 weight rows): group g owns
//               k-steps g, g + G_NG, ... It reads the row's 64 inputs of a k-step from the slot, de-quantises in
//               registers (int8 -> fp16 exactly; e2m1 x e4m3 block scale -> fp16 exactly) and writes them to tensor
//               memory (tcgen05.st: its 32 registers = 32 columns of its own TMEM lane), from where the MMA reads its
//               weight operand; shared memory carries the raw rows and the activation tiles.
//               One warp per scheduler cannot hide the latencies of this
//               serial instruction stream; several groups on different k-steps can. Afterwards all groups
//               run the epilogue: tcgen05.ld of 32 columns of their 32 TMEM lanes, row / tensor scale,
//               activation or residual; the fp16 tile is laid out in shared memory and leaves through TMA stores
//               (a residual tile comes in through TMA loads); products with a ragged row pitch store directly;
//   activation warp: TMA loads of the activation tile (tensor map over X, 128B swizzle);
//   MMA warp  : allocates TMEM; issues tcgen05.mma (kind::f16) and commits to mbarriers.
// Four-stage operand ring, all waits bounded (status word on expiry), TMEM freed on every path. Short grids with
// long K loops are split along K: every block of a tile finishes a share of its 32-row chunks, fetching the other
// blocks' fp32 partial sums of them from a scratch area with bulk copies and adding them in a fixed order. Launched with
// programmatic stream serialisation the kernel starts its weight stream before it waits for its predecessor.
//
// What bounds it: from 256 batch rows on the tensor core (a k-step of 320 rows takes 670 cycles of 640 at its rate); below
// that the memory and the hand-over between the warps, about 390 cycles a k-step whatever the batch (int8 rows at the
// copy bandwidth: 350). Around the main loop a block spends 1 us before it (tensor memory, barriers, first rows on their
// way) and 1 - 3 us behind it; the exchange of a split K costs 5 us.
// 16384 x 4096, back to back: 320 rows nvfp4 41.2 -> 35.4 us (1214 TFLOP/s), 64 rows nvfp4 32.0 -> 17.9 (24 rows int8 now 19.4),
// against the same kernel with cp.async rows and single-lane issue of MMAs and TMA copies (see *_one below). Launches of
// few rows, which none of this hides, go to stream.cu.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "gemm.cuh"
#include "gemv.cuh"

namespace ab {

namespace {

#ifndef G_NG_
#define G_NG_ 3
#endif
constexpr int G_NG = G_NG_;      // producer groups
constexpr int G_PROD = 128 * G_NG;
constexpr int GT = G_PROD + 128; // threads per block: producers + a warpgroup of the activation, MMA and weight warps and an idle one
                                 // (register re-allocation works on whole, aligned warpgroups)
#ifndef G_STAGES_
#define G_STAGES_ 4
#endif
constexpr int G_STAGES = G_STAGES_;
constexpr int G_A_COLS = 32;             // TMEM columns of one weight stage: 64 inputs as fp16 pairs
constexpr int G_BM = 128;        // weight rows per block
constexpr int G_BK = 64;         // inputs per k-step (128 bytes of fp16 = one swizzle row)
constexpr int G_RAW_ROW = 128;            // bytes of each weight row per raw slot: 1 / 2 / 4 k-steps of fp16 / int8 / NVFP4
constexpr int G_RAW_SLOTS = 12;           // at most this many raw slots
constexpr int G_REGS_PROD = 136, G_REGS_REST = 96;   // (136 - 128) * 384 producer threads <= (128 - 96) * 128 others
constexpr int G_MAX_OPS = 7;
constexpr int G_MAX_MAPS = 24;            // tensor maps of a launch
constexpr int G_COUNTERS = 4096;         // split-K arrival counters at the start of the scratch area

// One matrix product of a grouped launch.
struct GemmProb {
    ab_mat w;
    const __half* resid;
    __half* y;
    int epi;
    int ksplit;       // blocks that share one output tile along K
    int tile_base;    // first split-K tile id (counter / partial index)
    long long part_base;   // float offset of its split-K partial sums in the scratch area
    // which of the launch's tensor maps: activations X; weights as bytes, boxes of 128 rows x 128 bytes; NVFP4 block scales,
    // boxes of 128 rows x 16 bytes (-1: each thread loads its own); outputs Y and residuals, boxes of 32 batch rows x 128
    // features (-1: straight from and to global memory)
    signed char x_map, w_map, s_map, y_map, r_map;
    int recv_slots;   // split K: own chunks whose slices fit the receive area at a time
};
struct GemmGroup {
    int cta_base[G_MAX_OPS];   // first blockIdx.x of each product (unused ones: INT_MAX)
    GemmProb pr[G_MAX_OPS];
    int rows;       // batch rows (B*T)
    int n_tile;     // batch rows per block tile
    int n_first;    // batch rows of the first MMA of a k-substep (n_tile, or 192 when a second MMA takes the rest)
    int tma_rows;   // batch rows per TMA box
    int tmem_cols;
    int a_col0;     // first TMEM column of the weight stages (behind the accumulators)
    unsigned* counters;
    float* partials;
    int raw_bytes;  // shared memory for the raw slots
    int recv_off;   // split K: byte offset of the area the partial sums are fetched to, in the block's shared memory
};
// A launch with more than 4 KB of parameters costs the host more, so the maps share one table; products that find it full do
// without the optional ones. The host's part of an eager step of 12 blocks (61 launches of products): 283 us with five maps
// for every product (6 KB) and the weights' encoded for each launch, 256 like this; a prompt of 37 tokens 345 and 320.
struct GemmMaps {
    CUtensorMap t[G_MAX_MAPS];
};
static_assert(2 * G_MAX_OPS <= G_MAX_MAPS && sizeof(GemmMaps) + sizeof(GemmGroup) <= 4096, "parameters of the product kernels");

// ---------------------------------------------------------------------------------------------
// PTX wrappers (tcgen05 / TMA)
// ---------------------------------------------------------------------------------------------
// The wrappers named *_one are called by a whole, converged warp; one elected lane performs the operation. The election
// sits inside the assembly on purpose: an MMA issued from code that only one lane runs (`if (lane == 0)`) took 95 - 120
// cycles, timed by the kernel's own clock, which bounded every product here whatever its batch (a k-step of four: 480 cycles
// at 16 batch rows as at 192); elected like this it takes 34 (N <= 64) and runs at the tensor core's rate above (4 x N = 128:
// 257 cycles).
__device__ __forceinline__ void tma_load_2d_one(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n"
        " @q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n}" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_one(uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n @q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}" ::"r"(
                     smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y),
                 "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_drain_reads() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit_one(uint64_t* bar) {
    asm volatile(
        "{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(smem_u32(bar))
        : "memory");
}
// D (tensor memory) += A * B with the weight operand A read from tensor memory (128 lanes = weight rows, 8 columns = 16
// inputs as fp16 pairs) and the activations B from shared memory.
__device__ __forceinline__ void tc_mma_f16_one(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 registers of each of the warp's 32 lanes -> 32 consecutive TMEM columns of its 32 lanes.
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
          "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
          "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(G_PROD) : "memory"); }
__device__ __forceinline__ void group_sync(int grp) { asm volatile("bar.sync %0, 128;" ::"r"(2 + grp) : "memory"); }   // one producer group
constexpr int G_CHUNK_F32 = 32 * G_BM * 4;   // fp32 partial sums of 32 batch rows x 128 features

// K-major operand tile, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(const void* smem) {
    const uint32_t a = smem_u32(smem);
    uint64_t d = (uint64_t)((a >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;                 // leading byte offset: unused with swizzled K-major tiles
    d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                 // descriptor version of this architecture
    d |= (uint64_t)2 << 61;                 // SWIZZLE_128B
    return d;
}
// fp16 x fp16 -> fp32, both operands K-major, M = 128.
__device__ __forceinline__ uint32_t umma_idesc_f16(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(G_BM >> 4) << 24);
}

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__host__ __device__ constexpr int raw_ksteps(int fmt) { return fmt == FMT_I8 ? 2 : (fmt == FMT_FP4 ? 4 : 1); }   // k-steps per raw slot
__host__ __device__ constexpr int raw_slot_bytes(int fmt) { return G_BM * (G_RAW_ROW + (fmt == FMT_FP4 ? 16 : 0)); }

// 16-byte chunk c of row r of a raw slot (128-byte rows, 128-byte swizzle: eight consecutive rows, eight bank groups)
__device__ __forceinline__ uint4 raw_chunk(const unsigned char* slot, int r, int c) {
    return *reinterpret_cast<const uint4*>(slot + r * G_RAW_ROW + ((c ^ (r & 7)) << 4));
}
// De-quantise the 64 inputs of k-step `sub` of a raw slot for row r into eight 16-byte chunks of fp16 (chunk c =
// inputs 8c..8c+7): the raw bytes first (`raw`, so that the slot can be given back), then the arithmetic. Rows and
// inputs outside the matrix were zero-filled by the copy. sc4: NVFP4, the four block scales of these inputs.
template <int F>
__device__ __forceinline__ void raw_fetch(const unsigned char* slot, int r, int sub, uint4* raw) {
    constexpr int nq = 8 / raw_ksteps(F);
#pragma unroll
    for (int q = 0; q < nq; ++q) raw[q] = raw_chunk(slot, r, sub * nq + q);
}
template <int F>
__device__ __forceinline__ void raw_dequant(const uint4* raw, uint32_t sc4, uint4* out) {
    if (F == FMT_I8) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t words[4] = {raw[q].x, raw[q].y, raw[q].z, raw[q].w};
            uint32_t h[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                // int8 -> fp16 exactly: bytes b0, b1 into the mantissas of 1024 + (b ^ 0x80), then subtract 1152
                const uint32_t x = words[e] ^ 0x80808080u;
                const uint32_t lo = __byte_perm(x, 0x64646464u, 0x4140), hi = __byte_perm(x, 0x64646464u, 0x4342);
                const __half2 bias = __floats2half2_rn(1152.f, 1152.f);
                const __half2 l2 = __hsub2(*reinterpret_cast<const __half2*>(&lo), bias);
                const __half2 h2 = __hsub2(*reinterpret_cast<const __half2*>(&hi), bias);
                h[2 * e] = *reinterpret_cast<const uint32_t*>(&l2);
                h[2 * e + 1] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            out[2 * q] = make_uint4(h[0], h[1], h[2], h[3]);
            out[2 * q + 1] = make_uint4(h[4], h[5], h[6], h[7]);
        }
    } else if (F == FMT_F16) {
#pragma unroll
        for (int c = 0; c < 8; ++c) out[c] = raw[c];
    } else {
        const uint32_t words[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
        // the four block scales of these 64 inputs, each duplicated into both halves of a half2
        const __half2 s01 = e4m3x2_to_half2(sc4 & 0xffffu), s23 = e4m3x2_to_half2(sc4 >> 16);
        const __half2 scs[4] = {__low2half2(s01), __high2half2(s01), __low2half2(s23), __high2half2(s23)};
#pragma unroll
        for (int c = 0; c < 8; ++c) {   // chunk c: 8 inputs = 4 bytes; scale block = c / 2
            uint32_t h[4];
            e2m1x8_to_half2x4(words[c], h);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __half2 v = __hmul2(*reinterpret_cast<const __half2*>(&h[e]), scs[c >> 1]);   // exact in fp16
                h[e] = *reinterpret_cast<const uint32_t*>(&v);
            }
            out[c] = make_uint4(h[0], h[1], h[2], h[3]);
        }
    }
}

template <int EPI>
__device__ __forceinline__ float apply_epi_t(float o) {
    if (EPI == EPI_TANH) return tanhf(o);
    if (EPI == EPI_SIGMOID) return sigmoidf_(o);
    return o;
}
__device__ __forceinline__ float apply_epi(int epi, float o) {
    switch (epi) {
        case EPI_TANH: return tanhf(o);
        case EPI_SIGMOID: return sigmoidf_(o);
        case EPI_RELU2: o = fmaxf(o, 0.f); return o * o;
        default: return o;
    }
}

// SPLIT: some product of the launch is split along K (the lean instance is compiled without that ending).
// KS: k-steps per operand stage. The hand-over of a stage between the warps (waits, elections, commits) costs about 300
// cycles, an MMA of up to 64 batch rows 34: with up to 128 batch rows two k-steps share a hand-over (16384 x 4096, 8 rows
// int8: 22.0 -> 19.7 us, 128 rows: 23.9 -> 21.0). Taller tiles are bound by the tensor core and need the shared memory for
// the depth of the ring.
template <bool SPLIT, int KS>
__device__ __forceinline__ void gemm_block(const GemmMaps& maps, const GemmGroup& g) {
    extern __shared__ __align__(1024) unsigned char gsm[];
    constexpr int N_BARS = 2 * G_STAGES + 2 * G_RAW_SLOTS + 3;
    __shared__ uint64_t bars[N_BARS];
    uint64_t *full = bars, *empty = full + G_STAGES, *raw_full = empty + G_STAGES, *raw_empty = raw_full + G_RAW_SLOTS;
    uint64_t &accum_bar = bars[N_BARS - 3], &resid_bar = bars[N_BARS - 2], &recv_bar = bars[N_BARS - 1];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_failed;
    __shared__ uint32_t s_nobody;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 4 * G_NG + 1) tmem_alloc(&tmem_base_s, (uint32_t)g.tmem_cols);
    // ---- which product, which tile, which K split
    int pi = 0;
#pragma unroll
    for (int i = 1; i < G_MAX_OPS; ++i) pi += (int)blockIdx.x >= g.cta_base[i] ? 1 : 0;
    const GemmProb& pb = g.pr[pi];
    const int local = blockIdx.x - g.cta_base[pi];
    const bool split = SPLIT && pb.ksplit > 1;
    const int m_tile = split ? (int)((unsigned)local / (unsigned)pb.ksplit) : local, z = split ? local - m_tile * pb.ksplit : 0;
    const int m0 = m_tile * G_BM;
    const int n0 = blockIdx.y * g.n_tile;
    // K is dealt out in raw slots of `per` k-steps
    const int fmt = pb.w.fmt, per = raw_ksteps(fmt);
    const int total_ksteps = (pb.w.k + G_BK - 1) / G_BK, total_raw = (total_ksteps + per - 1) / per;
    const int raw_begin = split ? (int)((unsigned)total_raw * (unsigned)z / (unsigned)pb.ksplit) : 0;
    const int raw_end = split ? (int)((unsigned)total_raw * (unsigned)(z + 1) / (unsigned)pb.ksplit) : total_raw;
    const int n_raw = raw_end - raw_begin;
    const int n_ksteps = min(raw_end * per, total_ksteps) - raw_begin * per, n_stages = (n_ksteps + KS - 1) / KS;
    // Blocks walk K in rotated order: at any moment they read different columns of the (shared) activation
    // matrix, instead of all hitting the same few L2 lines. (Not where the last slot is only partly used: it comes last.)
    const int rot = total_ksteps % per ? 0 : (int)((blockIdx.x * 7u + blockIdx.y * 3u) % (unsigned)n_raw);
    auto raw_of = [&](int i) { int k = i + rot; if (k >= n_raw) k -= n_raw; return raw_begin + k; };   // i-th slot worked on
    const int slot_bytes = raw_slot_bytes(fmt);
    const int n_slots = min(G_RAW_SLOTS, g.raw_bytes / slot_bytes);

    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)gsm + 1023) & ~(uintptr_t)1023);
    const int tile_bytes = g.n_tile * 128, b_bytes = KS * tile_bytes;
    unsigned char* smB = base;                                  // G_STAGES x KS x n_tile x 128 B
    unsigned char* smRaw = smB + G_STAGES * b_bytes;            // raw weight slots

    if (tid < N_BARS) {
        // full: the four warps of the group that owns the stage + the activation warp's expect_tx; raw_empty: the four warps
        // of the owning group, for every stage that takes part of the slot
        const int i = tid - 2 * G_STAGES;
        mbar_init(&bars[tid], tid < G_STAGES ? 5u : (i >= G_RAW_SLOTS && i < 2 * G_RAW_SLOTS ? 4u * (unsigned)(per > KS ? per / KS : 1) : 1u));
        fence_mbar_init();
        if (tid == 0) s_failed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    // Registers go where the work is: the producers' de-quantisation needs more than an even share, the warps that only issue
    // copies and MMAs far less. (Whole warpgroups execute these: warps 0-3, 4-7, 8-11 / 12-15.)
    if (warp < 4 * G_NG) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(G_REGS_PROD));
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(G_REGS_REST));
    // Under programmatic stream serialisation the next grid may start now; like this one it begins with its weight
    // stream (weights are never written) and waits for its predecessor before it touches activations or outputs.
    if (tid == 0) pdl_launch_dependents();

    // After the first wait that runs out, nobody waits any more: the block drains in bounded time.
    auto wait_ok = [&](uint64_t* bar, uint32_t parity) {
        if (mbar_try_wait(bar, parity)) return;   // the common case costs one instruction
        if (*reinterpret_cast<volatile int*>(&s_failed)) return;
        if (!mbar_wait_bounded(bar, parity, 1u << 16)) {
            *reinterpret_cast<volatile int*>(&s_failed) = 1;
            atomicOr(&g_device_status, DEV_WAIT_GEMM);
        }
    };

    if (warp < 4 * G_NG) {
        // ===== weight producers: thread = weight row of the tile, group = every G_NG-th k-step =====
        const int grp = warp >> 2, r_local = tid & 127;
        const int row = m0 + r_local;
        const int n_out = pb.w.n_out;
        const bool row_ok = row < n_out;
        float scale = 1.f;   // of the output row; requested here, used in the epilogue
        if (row_ok) scale = fmt == FMT_I8 ? __ldg(reinterpret_cast<const float*>(pb.w.scale) + row) : pb.w.tscale;

        // One instance of the loop per weight format: chunk counts are constants in it, slots are walked with wrapping counters.
        auto produce = [&](auto fmt_c) {
            constexpr int F = decltype(fmt_c)::value;
            constexpr int P = raw_ksteps(F), SB = raw_slot_bytes(F);
            // block scales without a tensor map (k not a multiple of 256): this thread's own words, one own k-step ahead
            const bool own_sc = F == FMT_FP4 && pb.s_map < 0;
            const unsigned char* srow = reinterpret_cast<const unsigned char*>(pb.w.scale) + (F == FMT_FP4 && row_ok ? (size_t)row * (pb.w.k / 16) : 0);
            auto scale_word = [&](int ks) -> uint32_t {
                if (ks >= n_ksteps) return 0u;
                const int a = raw_of(ks / P) * P + ks % P;
                return row_ok && AB_BC(a >= 0 && a * 4 + 4 <= pb.w.k / 16) ? __ldg(reinterpret_cast<const unsigned*>(srow) + a) : 0u;
            };
            uint32_t sc_next = own_sc ? scale_word(grp * KS) : 0u;
            int slot = 0, sub = 0;
            uint32_t parity = 0;
            bool reused = false;   // the slot has held an earlier part of K
            auto advance = [&](int n) {
                sub += n;
                while (sub >= P) {
                    sub -= P;
                    if (++slot == n_slots) { slot = 0; parity ^= 1u; reused = true; }
                }
            };
            advance(grp * KS);
            int stage = grp % G_STAGES;
            uint32_t e_parity = 1;   // the first round finds every operand stage free
            for (int st = grp; st < n_stages; st += G_NG) {
#pragma unroll 1
                for (int h = 0; h < KS; ++h) {
                    const int ks = st * KS + h;
                    if (KS > 1 && ks >= n_ksteps) {   // an odd last k-step
                        if (P > 1 && lane == 0) mbar_arrive(&raw_empty[slot]);
                        break;
                    }
                    const unsigned char* raw_slot = smRaw + slot * SB;
                    uint32_t sc4 = sc_next;
                    if (own_sc) sc_next = scale_word(h < KS - 1 ? ks + 1 : ks + 1 + (G_NG - 1) * KS);
                    if (h == 0 || P == 1) {
                        // A slot's earlier content may have been another group's, and copies finish in any order: that copy
                        // may still be under way although this group's last one, issued after it, has landed. The phase bit
                        // alone cannot tell "two phases back" from "done", so first see that the earlier content has been
                        // used up. (Its copy had been issued by then - copies are issued in order and there are enough slots,
                        // see slots_suffice - so this wait is at most one phase back.)
                        if (reused) wait_ok(&raw_empty[slot], parity ^ 1u);
                        wait_ok(&raw_full[slot], parity);
                    }
                    uint4 raw[8 / P], cur[8];
                    raw_fetch<F>(raw_slot, r_local, sub, raw);
                    if (F == FMT_FP4 && !own_sc) sc4 = *reinterpret_cast<const uint32_t*>(raw_slot + G_BM * G_RAW_ROW + r_local * 16 + sub * 4);
                    if (h == KS - 1 || P == 1) {
                        uint32_t used = F == FMT_FP4 && !own_sc ? sc4 : 0u;
#pragma unroll
                        for (int q = 0; q < 8 / P; ++q) used ^= raw[q].x;
                        loads_returned(used, &s_nobody);
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&raw_empty[slot]);
                    }
                    raw_dequant<F>(raw, sc4, cur);
                    advance(1);
                    if (h == 0) {
                        if (st >= G_STAGES) wait_ok(&empty[stage], e_parity);
                        tc_fence_after();   // the MMAs that read this stage are complete (their commit released it)
                    }
                    // this thread's 64 inputs = 32 registers -> 32 columns of its own TMEM lane
                    tc_st32(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g.a_col0 + (stage * KS + h) * G_A_COLS),
                            reinterpret_cast<const uint32_t*>(cur));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[stage]);   // one arrival per warp of the owning group
                advance((G_NG - 1) * KS);
                stage += G_NG;
                if (stage >= G_STAGES) { stage -= G_STAGES; e_parity ^= 1u; }
            }
        };
        if (fmt == FMT_I8) produce(std::integral_constant<int, FMT_I8>());
        else if (fmt == FMT_FP4) produce(std::integral_constant<int, FMT_FP4>());
        else produce(std::integral_constant<int, FMT_F16>());
        pdl_wait();   // residuals and outputs belong to the preceding grids until here

        // ===== epilogue: thread = output feature (TMEM lane); groups take turns on chunks of 32 batch rows =====
        wait_ok(&accum_bar, 0);
        tc_fence_after();
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        const int n_valid = min(g.n_tile, g.rows - n0);
        const int n_chunks = (n_valid + 31) / 32;
        const int epi = pb.epi;

        // finished sums of 32 batch rows of this thread's feature -> fp16, stored straight to Y: the 32 lanes of a
        // warp write 32 consecutive features (64 bytes) of one batch row per instruction
        auto emit32 = [&](int ci, const float* v) {
            const int c0 = ci * 32;
            const size_t off = (size_t)(n0 + c0) * n_out + row;
            __half* yp = pb.y + off;
            if (!row_ok) return;
            if (epi == EPI_RESID) {
                const __half* rp = pb.resid + off;
#pragma unroll
                for (int h8 = 0; h8 < 32; h8 += 8) {   // eight loads in flight, then eight stores
                    __half rs[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) rs[i] = c0 + h8 + i < n_valid ? rp[(size_t)(h8 + i) * n_out] : __half(0.f);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (c0 + h8 + i < n_valid)
                            yp[(size_t)(h8 + i) * n_out] = __hadd(rs[i], __float2half_rn(v[h8 + i] * scale));
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (c0 + i < n_valid && AB_BC(row < n_out && n0 + c0 + i < g.rows)) yp[(size_t)i * n_out] = __float2half_rn(apply_epi(epi, rh(v[i] * scale)));
            }
        };

        // Preferred way out: the finished tile is laid out in shared memory as [batch row][128 features] fp16 (the
        // operand stages are idle by now) and leaves through the TMA unit in full lines; the unit clips rows and
        // features beyond the matrix. A residual tile comes in the same way and is updated in place.
        __half* stg = reinterpret_cast<__half*>(base);
        const bool staged = pb.y_map >= 0;
        auto stage32 = [&](int ci, const float* v) {
            __half* t = stg + (size_t)ci * 32 * G_BM + r_local;
            auto body = [&](auto E) {
                constexpr int EP = decltype(E)::value;
#pragma unroll
                for (int i = 0; i < 32; i += 2) {   // two batch rows at a time; the same roundings as one at a time
                    __half2 h = __floats2half2_rn(v[i] * scale, v[i + 1] * scale);
                    if (EP == EPI_RELU2) { h = __hmax2(h, __half2(__half(0.f), __half(0.f))); h = __hmul2(h, h); }
                    if (EP == EPI_RESID) h = __hadd2(__halves2half2(t[i * G_BM], t[(i + 1) * G_BM]), h);
                    if (EP == EPI_TANH || EP == EPI_SIGMOID) {
                        const float2 f = __half22float2(h);
                        h = __floats2half2_rn(apply_epi_t<EP>(f.x), apply_epi_t<EP>(f.y));
                    }
                    t[i * G_BM] = __low2half(h);
                    t[(i + 1) * G_BM] = __high2half(h);
                }
            };
            switch (epi) {
                case EPI_TANH: body(std::integral_constant<int, EPI_TANH>()); break;
                case EPI_SIGMOID: body(std::integral_constant<int, EPI_SIGMOID>()); break;
                case EPI_RELU2: body(std::integral_constant<int, EPI_RELU2>()); break;
                case EPI_RESID: body(std::integral_constant<int, EPI_RESID>()); break;
                default: body(std::integral_constant<int, EPI_NONE>()); break;
            }
        };
        // A staged chunk leaves at once, while the group works on its next chunk: the group's first thread hands it
        // to the TMA unit as soon as all four warps have written their part.
        auto emit = [&](int ci, const float* v) {
            if (!staged) { emit32(ci, v); return; }
            stage32(ci, v);
            fence_proxy_async();
            group_sync(grp);
            if (r_local == 0) {
                tma_store_2d(&maps.t[pb.y_map], m0, n0 + ci * 32, stg + (size_t)ci * 32 * G_BM);
                bulk_commit();
            }
        };
        // With split K every block of a tile finishes the chunks ci = z, z + ksplit, ... of it.
        auto my_chunk = [&](int ci) { return !split || ci % pb.ksplit == z; };
        // residual tiles on their way in
        auto fetch_resid = [&](bool wait = true) {
            if (!(staged && epi == EPI_RESID)) return;
            if (tid == 0) {
                int n_mine = 0;
                for (int ci = 0; ci < n_chunks; ++ci) n_mine += my_chunk(ci) ? 1 : 0;
                mbar_expect_tx(&resid_bar, (uint32_t)(n_mine * 32 * G_BM * 2));
                for (int ci = 0; ci < n_chunks; ++ci)
                    if (my_chunk(ci)) tma_load_2d(stg + (size_t)ci * 32 * G_BM, &maps.t[pb.r_map], m0, n0 + ci * 32, &resid_bar);
            }
            if (wait) wait_ok(&resid_bar, 0);
        };
        auto flush = [&]() {
            if (staged && r_local == 0) bulk_drain_reads();   // the shared memory must outlive the unit's reads
        };

        if (!split) {
            fetch_resid();
            for (int ci = grp; ci < n_chunks; ci += G_NG) {
                float v[32];
                tc_ld32(lane_addr + (uint32_t)(ci * 32), reinterpret_cast<uint32_t*>(v));
                emit(ci, v);
            }
            flush();
        } else {
            // Split K: chunk ci of the tile is finished by block ci % ksplit. Every block parks the partial sums of
            // the other blocks' chunks in the scratch area; once all blocks of the tile have done so, each fetches
            // the slices of its own chunks with bulk copies (all in flight at once) into the idle operand stages and
            // sums them in slice order (deterministic), its own slice coming from TMEM. The blocks of a tile wait
            // for one another: a split grid never has more blocks than the GPU has SMs and every block holds a
            // whole SM, so all of them are resident. The wait is bounded all the same.
            const int nz = pb.ksplit;
            const int tile = pb.tile_base + m_tile * gridDim.y + blockIdx.y;
            const size_t tile_floats = (size_t)g.n_tile * G_BM;
            float* tile0 = g.partials + pb.part_base + ((size_t)(m_tile * gridDim.y + blockIdx.y) * nz) * tile_floats;
            float* mine = tile0 + (size_t)z * tile_floats;
            fetch_resid(false);
            for (int ci = grp; ci < n_chunks; ci += G_NG) {
                if (ci % nz == z) continue;
                float v[32];
                tc_ld32(lane_addr + (uint32_t)(ci * 32), reinterpret_cast<uint32_t*>(v));
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (ci * 32 + i < g.n_tile) __stcg(mine + (size_t)(ci * 32 + i) * G_BM + r_local, v[i]);
            }
            __threadfence();
            epi_sync();
            bool ok = true;
            if (tid == 0) {
                atomicAdd(&g.counters[tile], 1u);
                uint32_t it = 0;
                while (ld_acquire_gpu(&g.counters[tile]) < (unsigned)nz) {
                    if (++it > (1u << 21)) {
                        ok = false;
                        atomicOr(&g_device_status, DEV_WAIT_GEMM);
                        break;
                    }
                }
                // the partial sums were written by ordinary stores of other blocks; the bulk copies read them
                asm volatile("fence.proxy.async;" ::: "memory");
            }
            if (staged && epi == EPI_RESID) wait_ok(&resid_bar, 0);
            unsigned char* recv = base + g.recv_off;
            const int n_own = z < n_chunks ? (n_chunks - z + nz - 1) / nz : 0;   // chunks z, z + nz, ...
            const int per_round = pb.recv_slots;   // own chunks whose slices fit the receive area at a time
            for (int k0 = 0, round = 0; k0 < n_own; k0 += per_round, ++round) {
                const int k1 = min(k0 + per_round, n_own);
                if (round > 0) epi_sync();   // everybody has read the slices of the round before
                if (tid == 0) {
                    uint32_t total = 0;
                    for (int kk = k0; kk < k1; ++kk)
                        total += (uint32_t)(nz - 1) * (uint32_t)(min(32, g.n_tile - (z + kk * nz) * 32) * G_BM * 4);
                    mbar_expect_tx(&recv_bar, ok ? total : 0u);
                    for (int kk = k0; ok && kk < k1; ++kk) {
                        const int ci = z + kk * nz;
                        const uint32_t bytes = (uint32_t)(min(32, g.n_tile - ci * 32) * G_BM * 4);
                        for (int zz = 0; zz < nz; ++zz) {
                            if (zz == z) continue;
                            bulk_g2s(recv + (size_t)((kk - k0) * (nz - 1) + (zz < z ? zz : zz - 1)) * G_CHUNK_F32,
                                     tile0 + (size_t)zz * tile_floats + (size_t)ci * 32 * G_BM, bytes, &recv_bar);
                        }
                    }
                }
                wait_ok(&recv_bar, (uint32_t)(round & 1));
                for (int kk = k0; kk < k1; ++kk) {
                    if (kk % G_NG != grp) continue;
                    const int ci = z + kk * nz;
                    float own[32], v[32];
                    tc_ld32(lane_addr + (uint32_t)(ci * 32), reinterpret_cast<uint32_t*>(own));
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = 0.f;
                    for (int zz = 0; zz < nz; ++zz) {
                        if (zz == z) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) v[i] += own[i];
                        } else {
                            const float* src = reinterpret_cast<const float*>(recv + (size_t)((kk - k0) * (nz - 1) + (zz < z ? zz : zz - 1)) * G_CHUNK_F32) + r_local;
#pragma unroll
                            for (int i = 0; i < 32; ++i) v[i] += src[i * G_BM];
                        }
                    }
                    emit(ci, v);
                }
            }
            flush();
            // the last block to leave puts the counter back to zero for the next launch
            if (tid == 0) {
                const unsigned old = atomicAdd(&g.counters[tile], 1u);
                if (old == 2u * (unsigned)nz - 1u) g.counters[tile] = 0;
            }
        }
        tc_fence_before();
    } else if (warp == 4 * G_NG) {
        // ===== activation tiles by TMA =====
        const CUtensorMap* map = &maps.t[pb.x_map];
        const bool two_boxes = g.tma_rows < g.n_tile;
        const int x_begin = raw_begin * per * G_BK, x_end = raw_end * per * G_BK;
        int x = raw_of(0) * per * G_BK;   // the k-steps in rotated order, walked without divisions
        uint32_t parity = 1;              // the first round finds every stage free
        pdl_wait();
        for (int st0 = 0; st0 < n_stages; st0 += G_STAGES, parity ^= 1u) {
#pragma unroll
            for (int s = 0; s < G_STAGES; ++s) {
                if (st0 + s >= n_stages) break;
                const int n_here = KS == 1 ? 1 : min(KS, n_ksteps - (st0 + s) * KS);
                if (st0 > 0) wait_ok(&empty[s], parity);
                __syncwarp();
                mbar_expect_tx_one(&full[s], (uint32_t)(n_here * tile_bytes));
#pragma unroll
                for (int h = 0; h < KS; ++h) {
                    if (h >= n_here) break;
                    unsigned char* dst = smB + s * b_bytes + h * tile_bytes;
                    tma_load_2d_one(dst, map, x, n0, &full[s]);
                    if (KS == 1 && two_boxes) tma_load_2d_one(dst + g.tma_rows * 128, map, x, n0 + g.tma_rows, &full[s]);
                    x += G_BK;
                    if (x == x_end) x = x_begin;
                }
            }
        }
    } else if (warp == 4 * G_NG + 2) {
        // ===== raw weights by TMA: never written by anybody, so they start before the preceding grid is done =====
        const uint32_t bytes = (uint32_t)(G_BM * G_RAW_ROW + (pb.s_map >= 0 ? G_BM * 16 : 0));
        const CUtensorMap *w_map = &maps.t[pb.w_map], *s_map = pb.s_map >= 0 ? &maps.t[pb.s_map] : nullptr;
        int slot = 0;
        uint32_t parity = 1;   // the first round finds every slot free
        for (int i = 0; i < n_raw; ++i) {
            if (i >= n_slots) wait_ok(&raw_empty[slot], parity);
            __syncwarp();
            unsigned char* dst = smRaw + slot * slot_bytes;
            const int ra = raw_of(i);
            mbar_expect_tx_one(&raw_full[slot], bytes);
            tma_load_2d_one(dst, w_map, ra * G_RAW_ROW, m0, &raw_full[slot]);
            if (s_map) tma_load_2d_one(dst + G_BM * G_RAW_ROW, s_map, ra * 16, m0, &raw_full[slot]);
            if (++slot == n_slots) { slot = 0; parity ^= 1u; }
        }
    } else if (warp == 4 * G_NG + 1) {
        // ===== MMA issue: the whole warp walks the loop, one elected lane issues =====
        // One lane feeds the tensor core, so its instruction stream is kept short: descriptors are built
        // once, a stage or a 16-input step further is an add to the (address >> 4) field.
        // An MMA is at most 256 batch rows wide and runs in steps of 64 of them: a 320-row tile is issued as
        // 192 + 128 on separate TMEM columns (160 + 160 would cost as much as 192 + 192).
        const uint32_t idesc = umma_idesc_f16(g.n_first);
        const uint64_t db0 = umma_desc_sw128(smB), b_stage = (uint64_t)(b_bytes >> 4);
        // unrolled over the stages: stage index, descriptors and barrier addresses are compile-time offsets
        auto issue = [&](auto two_c) {
            constexpr bool TWO = decltype(two_c)::value;
            const uint32_t idesc1 = TWO ? umma_idesc_f16(g.n_tile - g.n_first) : 0u, d1 = tmem_base + (uint32_t)g.n_first;
            const uint64_t b_half = (uint64_t)((g.n_first * 128) >> 4);
            uint32_t parity = 0;
            for (int st0 = 0; st0 < n_stages; st0 += G_STAGES, parity ^= 1u) {
#pragma unroll(KS == 1 ? G_STAGES : 1)
                for (int s = 0; s < G_STAGES; ++s) {
                    if (st0 + s >= n_stages) break;
                    const int n_here = KS == 1 ? 1 : min(KS, n_ksteps - (st0 + s) * KS);
                    wait_ok(&full[s], parity);
                    __syncwarp();
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < KS; ++h) {
                        if (h >= n_here) break;
                        const uint64_t db = db0 + (uint64_t)s * b_stage + (uint64_t)(h * (tile_bytes >> 4));
                        const uint32_t ta = tmem_base + (uint32_t)(g.a_col0 + (s * KS + h) * G_A_COLS);
#pragma unroll
                        for (int k4 = 0; k4 < G_BK / 16; ++k4) {   // 16 inputs = 8 columns of the weight stage, 32 bytes of the swizzle row
                            const uint32_t acc = h > 0 || k4 > 0 || s > 0 || st0 > 0 ? 1u : 0u;
                            tc_mma_f16_one(tmem_base, ta + (uint32_t)(8 * k4), db + (uint64_t)(2 * k4), idesc, acc);
                            if (TWO) tc_mma_f16_one(d1, ta + (uint32_t)(8 * k4), db + b_half + (uint64_t)(2 * k4), idesc1, acc);
                        }
                    }
                    tc_commit_one(&empty[s]);   // the stage may be refilled once these MMAs have read it
                }
            }
        };
        if (KS == 1 && g.n_first < g.n_tile) issue(std::true_type());
        else issue(std::false_type());
        tc_commit_one(&accum_bar);
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 4 * G_NG + 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)g.tmem_cols);
    }
}

template <bool SPLIT>
__global__ void __launch_bounds__(GT, 1) gemm_tc_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmGroup g) {
    gemm_block<SPLIT, 1>(maps, g);
}
template <bool SPLIT>
__global__ void __launch_bounds__(GT, 1) gemm_tc2_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmGroup g) {
    gemm_block<SPLIT, 2>(maps, g);
}

// In-register de-quantisation exactly as the product kernels do it, written out as fp32.
__global__ void dequant_kernel(ab_mat m, float* __restrict__ out) {
    const size_t total = (size_t)m.n_out * m.k;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int row = (int)(idx / m.k), col = (int)(idx % m.k);
        float v;
        if (m.fmt == FMT_I8) {
            v = (float)reinterpret_cast<const signed char*>(m.w)[idx] * reinterpret_cast<const float*>(m.scale)[row];
            if (m.col_scale) v *= m.col_scale[col];
        } else if (m.fmt == FMT_FP4) {
            const uint32_t byte = reinterpret_cast<const unsigned char*>(m.w)[idx >> 1];
            const float2 pr = __half22float2(e2m1x2_to_half2(byte));
            const float q = (col & 1) ? pr.y : pr.x;
            const float sb = e4m3_to_float(reinterpret_cast<const unsigned char*>(m.scale)[(size_t)row * (m.k / 16) + col / 16]);
            v = (q * sb) * m.tscale;
        } else {
            v = __half2float(reinterpret_cast<const __half*>(m.w)[idx]);
        }
        out[idx] = v;
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int get_encode_fn(EncodeTiledFn* out) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        AB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres));
        AB_CHECK_ARG(ptr && qres == cudaDriverEntryPointSuccess, "gemm: cuTensorMapEncodeTiled is not available");
        fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    *out = fn;
    return OK;
}

}  // namespace

int check_mat(const ab_mat& m, const char* what) {
    AB_CHECK_ARG(m.fmt == FMT_F16 || m.fmt == FMT_I8 || m.fmt == FMT_FP4, "%s: unknown weight format %d", what, m.fmt);
    AB_CHECK_ARG(m.w && m.n_out > 0 && m.k > 0, "%s: empty matrix", what);
    AB_CHECK_ARG(m.fmt == FMT_F16 || m.scale, "%s: scales missing", what);
    AB_CHECK_ARG(m.fmt != FMT_FP4 || m.k % 32 == 0, "%s: NVFP4 needs k %% 32 == 0", what);
    return OK;
}

int encode_weight_maps(const ab_mat& m, WeightMaps* out) {
    out->valid = out->scale_map = 0;
    if (!m.w || m.n_out <= 0 || m.k <= 0 || m.k % 16 != 0 || ((uintptr_t)m.w & 15) != 0 || (m.fmt == FMT_FP4 && (m.k % 64 != 0 || !m.scale)))
        return OK;
    EncodeTiledFn encode;
    const int st = get_encode_fn(&encode);
    if (st != OK) return st;
    // rows as they are stored; the block scales need a row pitch of a multiple of 16 bytes
    out->scale_map = m.fmt == FMT_FP4 && m.k % 256 == 0 && ((uintptr_t)m.scale & 15) == 0 ? 1 : 0;
    const cuuint32_t estr[2] = {1, 1};
    for (int which = 0; which < 1 + out->scale_map; ++which) {
        const cuuint64_t pitch = which ? m.k / 16 : (m.fmt == FMT_F16 ? 2ull * m.k : m.fmt == FMT_I8 ? (cuuint64_t)m.k : m.k / 2);
        const cuuint64_t wdim[2] = {pitch, (cuuint64_t)m.n_out};
        const cuuint32_t wbox[2] = {which ? 16u : (cuuint32_t)G_RAW_ROW, (cuuint32_t)G_BM};
        const CUresult cw = encode(which ? &out->s : &out->w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                                   const_cast<void*>(which ? m.scale : m.w), wdim, &pitch, wbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   which ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cw != CUDA_SUCCESS) {
            set_error("gemm: cuTensorMapEncodeTiled (weights) failed with %d (n_out=%d k=%d fmt=%d)", (int)cw, m.n_out, m.k, m.fmt);
            return ERR_CUDA;
        }
    }
    out->valid = 1;
    return OK;
}

namespace {

struct GroupShape {
    int n_tile, n_first, tma_rows, tmem_cols, n_tiles_y;
    int ksplit[G_MAX_OPS];
    int grid_x;
    long long part_floats;
    int n_split_tiles;
};

// Shared memory of a block (beyond the 1 KB alignment slack): a block owns its SM (registers), so it takes all of it.
constexpr int G_SMEM = 225 * 1024;
// k-steps per operand stage (see gemm_block) and what the stages leave for the raw weight slots.
constexpr int stage_ksteps(int n_tile) { return n_tile <= 128 ? 2 : 1; }
constexpr int raw_smem(int n_tile) { return G_SMEM - G_STAGES * stage_ksteps(n_tile) * n_tile * 128; }
// What the phase bits of the slots rely on (see the wait in gemm_block): when a producer group comes to a k-step, the copy
// that filled its slot the time before has been issued. Copies are issued in order, so that holds if there are at least as
// many slots as lie between two k-steps that the group visits one after the other. The tallest tiles leave the fewest: 320
// rows 4 slots (fp16: 3 needed, int8: 2) or 3 (NVFP4 with its scales: 1), 128 rows, two k-steps a stage, 6 (5, 3) or 5 (2).
constexpr bool slots_suffice(int fmt, int n_tile) {
    const int ks = stage_ksteps(n_tile), apart = G_NG * ks - (ks - 1), per = raw_ksteps(fmt);
    return raw_smem(n_tile) / raw_slot_bytes(fmt) >= (apart + per - 1) / per;
}
static_assert(slots_suffice(FMT_F16, 320) && slots_suffice(FMT_I8, 320) && slots_suffice(FMT_FP4, 320) && slots_suffice(FMT_F16, 128) &&
                  slots_suffice(FMT_I8, 128) && slots_suffice(FMT_FP4, 128),
              "too few raw weight slots for this number of operand stages and producer groups");
// Split K: how many of its own chunks a block can fetch the other blocks' partial sums for at a time. They land
// in the operand stages behind the output staging area.
int split_recv_slots(int n_tile, int ks) {
    const int n_chunks = (n_tile + 31) / 32;
    const size_t stage_bytes = (size_t)n_chunks * 32 * G_BM * 2;
    const size_t avail = G_SMEM - stage_bytes;
    const int own_max = (n_chunks + ks - 1) / ks;
    const int fit = (int)(avail / ((size_t)(ks - 1) * G_CHUNK_F32));
    return fit < own_max ? fit : own_max;
}

// tall_tile: the batch rows per tile for more rows than one tile holds.
GroupShape group_shape(const GemmOp* ops, int n, int rows, int n_sm, int tall_tile) {
    GroupShape gs = {};
    if (rows <= 256) { gs.n_tile = (rows + 15) & ~15; gs.n_first = gs.tma_rows = gs.n_tile; }
    else if (rows <= 320) { gs.n_tile = (rows + 31) & ~31; gs.n_first = 192; gs.tma_rows = gs.n_tile / 2; }
    else {
        gs.n_tile = gs.n_first = gs.tma_rows = tall_tile;
        if (gs.n_tile > 256) { gs.n_first = 192; gs.tma_rows = gs.n_tile / 2; }
    }
    gs.tmem_cols = 32;
    const int a_cols = G_STAGES * stage_ksteps(gs.n_tile) * G_A_COLS;   // weight stages behind the accumulators
    while (gs.tmem_cols < ((gs.n_tile + 31) & ~31) + a_cols) gs.tmem_cols *= 2;
    gs.n_tiles_y = (rows + gs.n_tile - 1) / gs.n_tile;
    int base_ctas = 0, slow_ctas = 0;
    for (int i = 0; i < n; ++i) {
        const int c = (ops[i].w.n_out + G_BM - 1) / G_BM * gs.n_tiles_y;
        base_ctas += c;
        if (ops[i].w.fmt == FMT_F16 && ops[i].w.k >= 32 * G_BK) slow_ctas += c;
    }
    for (int i = 0; i < n; ++i) {
        const int ksteps = (ops[i].w.k + G_BK - 1) / G_BK;
        int ks = 1;
        if (base_ctas > 0 && base_ctas < (100 * n_sm) / 148 && ksteps >= 32) {   // too few tiles to fill the GPU: split the long K loops
            ks = n_sm / base_ctas;
            if (ks > 8) ks = 8;
            if (ks > ksteps / 8) ks = ksteps / 8;
            if (ks < 1) ks = 1;
        } else if (base_ctas < n_sm && slow_ctas > 0 && ops[i].w.fmt == FMT_F16 && ksteps >= 32) {
            // A nearly full grid whose fp16 products move two to four times the bytes per k-step of the quantised ones: they
            // would finish last, and the idle SMs take slices of their K loops. A step of two blocks, 4096 wide, with and
            // without (us): int8 100 rows 324, 333; 320 rows 621, 644; nvfp4 64 rows 281, 285; 320 rows 603, 620; all fp16 up to
            // 160 rows alike, 320 rows 664, 676.
            ks = 1 + (n_sm - base_ctas) / slow_ctas;
            if (ks > 8) ks = 8;
            if (ks > ksteps / 8) ks = ksteps / 8;
            if (ks < 1) ks = 1;
        }
        while (ks > 1 && split_recv_slots(gs.n_tile, ks) < 1) --ks;   // the slices of one chunk must fit the receive area
        gs.ksplit[i] = ks;
        const int m_tiles = (ops[i].w.n_out + G_BM - 1) / G_BM;
        gs.grid_x += m_tiles * ks;
        if (ks > 1) {
            gs.part_floats += (long long)m_tiles * gs.n_tiles_y * ks * gs.n_tile * G_BM;
            gs.n_split_tiles += m_tiles * gs.n_tiles_y;
        }
    }
    return gs;
}

// The shape a launch runs with. For more than 320 rows the tile height is a choice: fewer, taller tiles read the weights fewer
// times and may be split along K, more and lower ones fill the SMs without an exchange. A block's time is its k-steps times
// what one costs (420 cycles up to 128 rows, where two share a hand-over; above, the tensor core's 2.1 per row, 450 at least)
// plus what surrounds them; a launch takes as many of those as there are rounds of blocks over the SMs, and the exchange where
// it is split. The height with the smallest sum; over 96 products of 400 - 768 rows that is within 10 % of the fastest and level
// with it on average. 400 rows, int8, a fixed tile of 256, this rule, and one that leaves the split out: 4096 x 4096 inputs 22.9, 21.1
// (128 rows), 20.8 us; 2560 x 10240 inputs 29.8, 28.9 (224 rows, three ways), 38.8 (128 rows, 80 blocks of 160 k-steps).
// A height whose partial sums need more scratch than 256 rows do is left out: what a caller's scratch area has to hold, and
// which products the built-in one takes, does not depend on the choice.
constexpr int G_TALL = 256;
GroupShape launch_shape(const GemmOp* ops, int n, int rows, int n_sm) {
    const GroupShape ref = group_shape(ops, n, rows, n_sm, G_TALL);
    if (rows <= 320) return ref;
    const int sms = n_sm > 0 ? n_sm : 148;
    GroupShape pick = ref;
    long long best = 0;
    for (int t = 320; t >= 128; t -= 32) {   // whole 32-row chunks: the next tile's rows are not this one's to store
        const GroupShape gs = t == G_TALL ? ref : group_shape(ops, n, rows, n_sm, t);
        if (gs.part_floats > ref.part_floats) continue;
        int ksteps = 1;
        for (int i = 0; i < n; ++i) ksteps = std::max(ksteps, ((ops[i].w.k + G_BK - 1) / G_BK + gs.ksplit[i] - 1) / gs.ksplit[i]);
        const int rounds = (gs.grid_x * gs.n_tiles_y + sms - 1) / sms, per_step = t <= 128 ? 420 : std::max(450, 21 * t / 10);
        const long long cost = rounds * ((long long)ksteps * per_step + 6000 + 30 * t) + (gs.n_split_tiles ? 4000 + 30 * t : 0);
        if (best == 0 || cost < best) { best = cost; pick = gs; }
    }
    return pick;
}

}  // namespace

// SMs of the current device (148 on B200); the split-K decisions depend on it.
int current_sm_count() {
    static PerDeviceOnce once;
    const DeviceProps* dp = nullptr;
    if (once.run(&dp, [](DeviceProps&) -> int { return OK; }) != OK || !dp || dp->n_sm <= 0) return 148;
    return dp->n_sm;
}

size_t gemm_group_scratch_bytes(const GemmOp* ops, int n, int rows) {
    if (!ops || n < 1 || n > G_MAX_OPS || rows <= 0) return 0;
    for (int i = 0; i < n; ++i)
        if (ops[i].w.n_out <= 0 || ops[i].w.k <= 0) return 0;
    // (launch_shape never takes more)
    return (size_t)G_COUNTERS * 4 + (size_t)group_shape(ops, n, rows, current_sm_count(), G_TALL).part_floats * 4 + 256;
}
size_t gemm_scratch_bytes(const ab_mat& m, int rows) {
    GemmOp op = {};
    op.w = m;
    return gemm_group_scratch_bytes(&op, 1, rows);
}

int gemm_group_launch(const GemmOp* ops, int n, int rows, void* scratch, size_t scratch_bytes, cudaStream_t stream, bool pdl) {
    AB_CHECK_ARG(ops && n >= 1 && n <= G_MAX_OPS && rows > 0, "gemm: bad group (n=%d rows=%d)", n, rows);
    for (int i = 0; i < n; ++i) {   // shapes first: the grid arithmetic below divides by tile counts
        const int s = check_mat(ops[i].w, "gemm");
        if (s != OK) return s;
    }
    int st = OK;
    for (int i = 0; i < n; ++i) {
        const GemmOp& op = ops[i];
        const ab_mat& m = op.w;
        AB_CHECK_ARG(op.x && op.y, "gemm: null activation pointer");
        AB_CHECK_ARG(op.epi >= EPI_NONE && op.epi <= EPI_RESID && (op.epi != EPI_RESID || op.resid), "gemm: bad epilogue");
        AB_CHECK_ARG(m.col_scale == nullptr, "gemm: per-input-column scales are a batch-1 feature");
        AB_CHECK_ARG(m.k % 16 == 0 && ((uintptr_t)op.x & 15) == 0 && ((uintptr_t)m.w & 15) == 0, "gemm: k %% 16 and 16-byte alignment needed");
        AB_CHECK_ARG(m.fmt != FMT_FP4 || (m.k % 64 == 0 && ((uintptr_t)m.scale & 3) == 0), "gemm: NVFP4 needs k %% 64 == 0");
    }
    // few rows: before the split of this kernel is planned (a prompt of 2 to 24 tokens plans every launch anew); a call
    // without a scratch area is refused below where this kernel would need one, whichever kernel would run
    const bool has_scratch = scratch && ((uintptr_t)scratch & 15) == 0;
    bool taken = false;
    if (has_scratch) {
        st = stream_group_launch(ops, n, rows, stream, pdl, &taken);
        if (st != OK || taken) return st;
    }
    const int n_sm = current_sm_count();
    GroupShape gs = launch_shape(ops, n, rows, n_sm);
    AB_CHECK_ARG(gs.n_split_tiles <= G_COUNTERS, "gemm: too many split-K tiles");
    if (gs.n_split_tiles > 0 && (gs.grid_x * gs.n_tiles_y > n_sm || (size_t)G_COUNTERS * 4 + (size_t)gs.part_floats * 4 > scratch_bytes)) {
        // the blocks of a split tile wait for one another, so all of them must be resident (one block per SM), and their
        // partial sums must fit the scratch area; a split grid for which that does not hold is launched without the split
        GemmOp unsplit[G_MAX_OPS];
        for (int i = 0; i < n; ++i) unsplit[i] = ops[i];
        gs = launch_shape(unsplit, n, rows, 0);   // no SMs to fill: every product keeps its whole K loop
    }
    AB_CHECK_ARG(gs.part_floats == 0 || has_scratch, "gemm: split-K needs a 16-byte aligned scratch area");
    if (!has_scratch) {
        st = stream_group_launch(ops, n, rows, stream, pdl, &taken);
        if (st != OK || taken) return st;
    }
    EncodeTiledFn encode;
    st = get_encode_fn(&encode);
    if (st != OK) return st;

    GemmGroup g = {};
    GemmMaps maps;
    g.rows = rows; g.n_tile = gs.n_tile; g.n_first = gs.n_first; g.tma_rows = gs.tma_rows; g.tmem_cols = gs.tmem_cols;
    g.a_col0 = (gs.n_tile + 31) & ~31;
    g.raw_bytes = raw_smem(gs.n_tile);
    g.recv_off = (gs.n_tile + 31) / 32 * 32 * G_BM * 2;
    g.counters = reinterpret_cast<unsigned*>(scratch);
    g.partials = scratch ? reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(scratch) + (size_t)G_COUNTERS * 4) : nullptr;
    int cta = 0, tile = 0, n_maps = 0;
    long long part = 0;
    for (int i = 0; i < n; ++i) {
        const GemmOp& op = ops[i];
        const ab_mat& m = op.w;
        GemmProb& pb = g.pr[i];
        pb.w = m; pb.resid = op.resid; pb.y = op.y; pb.epi = op.epi;
        g.cta_base[i] = cta; pb.ksplit = gs.ksplit[i]; pb.tile_base = tile; pb.part_base = part;
        pb.recv_slots = pb.ksplit > 1 ? split_recv_slots(gs.n_tile, pb.ksplit) : 0;
        const int m_tiles = (m.n_out + G_BM - 1) / G_BM;
        cta += m_tiles * pb.ksplit;
        if (pb.ksplit > 1) {
            tile += m_tiles * gs.n_tiles_y;
            part += (long long)m_tiles * gs.n_tiles_y * pb.ksplit * gs.n_tile * G_BM;
        }
        const cuuint64_t gdim[2] = {(cuuint64_t)m.k, (cuuint64_t)rows};
        const cuuint64_t gstride[1] = {(cuuint64_t)m.k * 2};
        const cuuint32_t box[2] = {(cuuint32_t)G_BK, (cuuint32_t)gs.tma_rows};
        const cuuint32_t estr[2] = {1, 1};
        const CUresult cr = encode(&maps.t[pb.x_map = (signed char)n_maps++], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(op.x), gdim, gstride, box,
                                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) {
            set_error("gemm: cuTensorMapEncodeTiled failed with %d (rows=%d k=%d)", (int)cr, rows, m.k);
            return ERR_CUDA;
        }
        WeightMaps own;
        const WeightMaps* wm = op.maps && op.maps->valid ? op.maps : &own;
        if (wm == &own) {
            st = encode_weight_maps(m, &own);
            if (st != OK) return st;
        }
        maps.t[pb.w_map = (signed char)n_maps++] = wm->w;
        // (the obligatory maps of the products behind this one keep their places)
        const int room = G_MAX_MAPS - n_maps - 2 * (n - 1 - i);
        pb.s_map = pb.y_map = pb.r_map = -1;
        // output / residual tiles through the TMA unit when the row pitch and the pointers allow it
        const int out_maps = op.epi == EPI_RESID ? 2 : 1;
        if (m.n_out % 8 == 0 && m.n_out >= G_BM && ((uintptr_t)op.y & 15) == 0 && (op.epi != EPI_RESID || ((uintptr_t)op.resid & 15) == 0) &&
            out_maps <= room) {
            pb.y_map = (signed char)n_maps++;
            if (op.epi == EPI_RESID) pb.r_map = (signed char)n_maps++;
            const cuuint64_t odim[2] = {(cuuint64_t)m.n_out, (cuuint64_t)rows};
            const cuuint64_t ostride[1] = {(cuuint64_t)m.n_out * 2};
            const cuuint32_t obox[2] = {(cuuint32_t)G_BM, 32};
            CUresult c2 = encode(&maps.t[pb.y_map], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, op.y, odim, ostride, obox, estr,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (c2 == CUDA_SUCCESS && op.epi == EPI_RESID)
                c2 = encode(&maps.t[pb.r_map], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(op.resid), odim, ostride, obox,
                            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (c2 != CUDA_SUCCESS) {
                set_error("gemm: cuTensorMapEncodeTiled (output) failed with %d (rows=%d n_out=%d)", (int)c2, rows, m.n_out);
                return ERR_CUDA;
            }
        }
        if (wm->scale_map && (pb.y_map < 0 ? room : room - out_maps) > 0) maps.t[pb.s_map = (signed char)n_maps++] = wm->s;
    }
    for (int i = n; i < G_MAX_OPS; ++i) g.cta_base[i] = 0x7fffffff;

    const size_t smem = 1024 + G_SMEM;
    {
        static PerDeviceOnce once;
        const int s = once.run(nullptr, [](DeviceProps& d) -> int {
            // the largest dynamic size the device allows (the kernels' static shared memory is under 1 KB)
            for (auto k : {gemm_tc_kernel<false>, gemm_tc_kernel<true>, gemm_tc2_kernel<false>, gemm_tc2_kernel<true>})
                AB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d.smem_optin - 1024));
            return OK;
        });
        if (s != OK) return s;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gs.grid_x, gs.n_tiles_y);
    cfg.blockDim = dim3(GT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (pdl) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    const bool two = stage_ksteps(gs.n_tile) == 2, any_split = gs.n_split_tiles > 0;
    AB_CUDA(cudaLaunchKernelEx(&cfg, two ? (any_split ? gemm_tc2_kernel<true> : gemm_tc2_kernel<false>)
                                         : (any_split ? gemm_tc_kernel<true> : gemm_tc_kernel<false>), maps, g));
    return OK;
}

int gemm_launch(const ab_mat& m, int rows, const __half* x, __half* y, int epi, const __half* resid, void* scratch,
                size_t scratch_bytes, cudaStream_t stream, bool pdl, const WeightMaps* maps) {
    GemmOp op = {};
    op.w = m; op.x = x; op.y = y; op.epi = epi; op.resid = resid; op.maps = maps;
    return gemm_group_launch(&op, 1, rows, scratch, scratch_bytes, stream, pdl);
}

int dequant_launch(const ab_mat& m, float* out, cudaStream_t stream) {
    int s = check_mat(m, "dequant");
    if (s != OK) return s;
    AB_CHECK_ARG(out, "dequant: null output");
    dequant_kernel<<<1184, 256, 0, stream>>>(m, out);
    AB_CUDA(cudaGetLastError());
    return OK;
}

}  // namespace ab

// ---------------------------------------------------------------------------------------------
// Batched product with built-in scratch: the split-K counters and partial tiles live in a fixed array of this
// module instead of a caller-supplied buffer, so the call neither takes nor makes a device allocation.
// ---------------------------------------------------------------------------------------------
namespace ab {
namespace {

static __device__ __align__(256) unsigned char g_static_scratch[AB_GEMM_STATIC_SCRATCH_BYTES];

constexpr int STATIC_MAX_DEVICES = AB_MAX_DEVICES;
std::mutex g_static_mu;
void* g_static_ptrs[STATIC_MAX_DEVICES] = {};

// Address of the array on the current device, looked up once per device (under a lock: the first calls of two host
// threads may coincide); the counters are cleared on `stream` when a device is first used (the kernels need them at
// zero and leave them at zero).
int static_scratch(void** out, cudaStream_t stream) {
    int dev = 0;
    AB_CUDA(cudaGetDevice(&dev));
    AB_CHECK_ARG(dev >= 0 && dev < STATIC_MAX_DEVICES, "ab_gemm_static: device index %d not supported", dev);
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptrs[dev]) {
        void* ptr = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || !ptr) {
            set_error("ab_gemm_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return ERR_CUDA;
        }
        AB_CUDA(cudaMemsetAsync(ptr, 0, (size_t)G_COUNTERS * 4, stream));
        g_static_ptrs[dev] = ptr;
    }
    *out = g_static_ptrs[dev];
    return OK;
}

}  // namespace

// Puts the arrival counters of the built-in scratch area of the current device back to zero (nothing to do if the
// device has not used it yet). The kernels leave them at zero themselves, except when a bounded wait gave up or a
// launch was aborted half-way; then every later split-K product through ab_gemm_static would read stale counts.
int static_scratch_reset(cudaStream_t stream) {
    int dev = 0;
    AB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= STATIC_MAX_DEVICES) return OK;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (g_static_ptrs[dev]) AB_CUDA(cudaMemsetAsync(g_static_ptrs[dev], 0, (size_t)G_COUNTERS * 4, stream));
    return OK;
}

}  // namespace ab

extern "C" int ab_gemm_plan_selftest(const int32_t* fmt, const int32_t* n_out, const int32_t* k, int n, int rows, int n_sm, int32_t* tile,
                                     int32_t* blocks, int32_t* ksplit) {
    using namespace ab;
    AB_CHECK_ARG(fmt && n_out && k && tile && blocks && ksplit && n >= 1 && n <= G_MAX_OPS && rows > 0 && n_sm >= 0, "ab_gemm_plan_selftest: bad argument");
    GemmOp ops[G_MAX_OPS] = {};
    for (int i = 0; i < n; ++i) {
        AB_CHECK_ARG(n_out[i] > 0 && k[i] > 0, "ab_gemm_plan_selftest: empty matrix");
        ops[i].w.fmt = fmt[i]; ops[i].w.n_out = n_out[i]; ops[i].w.k = k[i];
    }
    const GroupShape gs = launch_shape(ops, n, rows, n_sm), ref = group_shape(ops, n, rows, n_sm, G_TALL);
    AB_CHECK_ARG(gs.part_floats <= ref.part_floats, "ab_gemm_plan_selftest: %lld partial sums, scratch for %lld", gs.part_floats, ref.part_floats);
    AB_CHECK_ARG(gs.n_split_tiles == 0 || gs.grid_x * gs.n_tiles_y <= n_sm, "ab_gemm_plan_selftest: %d blocks of a split grid", gs.grid_x * gs.n_tiles_y);
    AB_CHECK_ARG(gs.n_tiles_y * gs.n_tile >= rows && (gs.n_tiles_y == 1 || gs.n_tile % 32 == 0), "ab_gemm_plan_selftest: tiles of %d rows", gs.n_tile);
    *tile = gs.n_tile;
    *blocks = gs.grid_x * gs.n_tiles_y;
    for (int i = 0; i < n; ++i) ksplit[i] = gs.ksplit[i];
    return OK;
}

extern "C" int ab_gemm_static(const ab_mat* m, int rows, const void* x, void* y, int epi, const void* resid, void* stream) {
    using namespace ab;
    AB_CHECK_ARG(m && x && y, "ab_gemm_static: null pointer");
    AB_CHECK_ARG(epi >= EPI_NONE && epi <= EPI_RESID && (epi != EPI_RESID || resid), "ab_gemm_static: bad epilogue");
    AB_CHECK_ARG(rows > 0, "ab_gemm_static: rows must be positive");
    int st = check_mat(*m, "ab_gemm_static");
    if (st != OK) return st;
    const size_t need = gemm_scratch_bytes(*m, rows);
    if (need > (size_t)AB_GEMM_STATIC_SCRATCH_BYTES) {
        set_error("ab_gemm_static: this product needs %zu bytes of split-K scratch, the built-in area holds %zu "
                  "(n_out=%d k=%d rows=%d); use ab_gemm with a caller-supplied scratch buffer",
                  need, (size_t)AB_GEMM_STATIC_SCRATCH_BYTES, m->n_out, m->k, rows);
        return ERR_TOO_LARGE;
    }
    void* scratch = nullptr;
    st = static_scratch(&scratch, (cudaStream_t)stream);
    if (st != OK) return st;
    return gemm_launch(*m, rows, (const __half*)x, (__half*)y, epi, (const __half*)resid, scratch, (size_t)AB_GEMM_STATIC_SCRATCH_BYTES,
                       (cudaStream_t)stream);
}

extern "C" int ab_gemm_static_reset(void* stream) { return ab::static_scratch_reset((cudaStream_t)stream); }

// Test hook: reads (write == 0) or overwrites (write != 0) arrival counter `index` of the built-in scratch area of the
// current device, through `value_host`. Synchronises the device.
extern "C" int ab_gemm_static_debug_counter(int index, int write, uint32_t* value_host) {
    using namespace ab;
    AB_CHECK_ARG(value_host && index >= 0 && index < G_COUNTERS, "ab_gemm_static_debug_counter: bad argument");
    void* scratch = nullptr;
    const int st = static_scratch(&scratch, nullptr);
    if (st != OK) return st;
    AB_CUDA(cudaDeviceSynchronize());
    uint32_t* p = reinterpret_cast<uint32_t*>(scratch) + index;
    if (write) AB_CUDA(cudaMemcpy(p, value_host, 4, cudaMemcpyHostToDevice));
    else AB_CUDA(cudaMemcpy(value_host, p, 4, cudaMemcpyDeviceToHost));
    return OK;
}


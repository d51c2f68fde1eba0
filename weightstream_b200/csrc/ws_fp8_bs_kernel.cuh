// FP8 E4M3 row-parallel GEMM on the 5th-generation tensor cores with block scaling
// (tcgen05.mma.kind::mxf8f6f4.block_scale, accumulators in tensor memory), fused with its
// exchange (sm_100a).  One pass over the weights for up to 128 activation rows.
//
//   act_prep_kernel   quantises the activations once per step exactly as the reference does
//                     (crates/weightstream-ref/src/actquant.rs:21-57) into the form the MMA reads: 16-byte
//                     chunks of K, chunk-major ([chunk][token][16 bytes]), and the per-32 exponents as one
//                     scale atom per 128-wide K slab.
//   fp8_bs_kernel     persistent, one CTA per SM.  The rows are cut into tiles of at most 128 rows (the
//                     M of the MMA), dealt out whole; a CTA (or a CTA pair, each CTA one half of K)
//                     streams the weights of its tiles, so every output is a complete dot product inside
//                     one CTA pair and nothing is combined through global memory.  A stage of the ring
//                     holds SL K slabs of 128: their weight rows (a TMA box each, 128B swizzle), their
//                     activations and their scale atoms (one bulk copy).  The activation operand is
//                     unswizzled K-major with core matrices 16 * m bytes apart along K, so m tokens take
//                     m * 128 bytes per slab whatever N is: its columns past m read the neighbouring chunk
//                     and are never looked at.  (Padded to N rows the activations of 40 tokens were as many
//                     bytes as the weights, and what L2 can hand the SMs bound the step.)  An atom is
//                     min(m, 32) rows of 16 bytes: byte (t & 31) * 16 + (t >> 5) * 4 + j = exponent of token
//                     t, K block j.
//                     INL: up to 8192 values per CTA its epilogue warps quantise them straight into shared memory
//                     and there is no prep launch.
//                     One thread copies the atoms into tensor memory (tcgen05.cp) and issues four MMAs per
//                     slab (M=128, N=tokens, K=32): the activations' per-32 scales ride the MMA's scale
//                     operand.
//   Weight scales     fp32 per (block_n x block_k) fit no MMA scale format: the weight operand's scale is
//                     2^0, every slab has its own accumulator buffer, and the epilogue warps read a stage's
//                     buffers back (tcgen05.ld) and add them x the fp32 scale while later MMAs run.
//                     UE8M0 (WUE): they ARE an MMA scale operand.  Four auxiliary warps lay the tile's scale
//                     bytes out as atoms in the stage; an accumulator takes two slabs (see bs_chain).
//
// Measured on B200 and kept in mind above: every TMA or bulk copy costs its issuing thread 85-100 ns, but
// one 3-D box for a stage's slabs was slower than a box each (128 rows 32.0 against 29.4 us); a slab's four
// MMAs, scale copy and share of the commit take the tensor pipe 84 ns with N=16, 105 with 64 and 135 with 128,
// however few of the 128 rows are real (M=64 is not available with block scaling); handing partial sums from one
// CTA to another through L2 (a split of K across CTAs) costs 3-5 us, more than it saves on these shapes.
//
// MMA rows past a tile's end are computed on whatever follows in shared memory and never read back.
// Exchange and lm_head mode are those of the decode kernels (ws_fp8_kernel.cuh): tagged 64-bit
// words stored into every peer's slots and folded in rank order, or logits gathered and argmax candidates
// merged per rank.
#pragma once

#include <math.h>

#include <type_traits>

#include "ws_device.cuh"
#include "ws_fp8_kernel.cuh"

namespace ws {

// Threads of a CTA.  Warp 0: producer, warp 1: MMA issue (and owner of the tensor memory), then the
// epilogue warps: four (one per 32-lane quarter of the tensor memory, all token columns) for up to 16
// tokens, eight (two per quarter, half of the token columns each) beyond, where reading the
// accumulators back is what a stage waits for (sixteen for 128 tokens: 38 against 31 us); then, for UE8M0
// weight scales, four auxiliary warps.
__host__ __device__ constexpr int bs_epi_warps(int mp) { return mp >= 32 ? 8 : 4; }
constexpr int kBsAuxWarps = 4;
__host__ __device__ constexpr int bs_threads(int mp, bool wue) { return 64 + 32 * (bs_epi_warps(mp) + (wue ? kBsAuxWarps : 0)); }
// Registers per thread: what leaves a warp of the prep kernel room in every quarter of the SM's register file
// (a CTA of ten warps has three in two of them, one of fourteen has four; the next step's prep blocks otherwise wait
// for the CTA to leave: UE8M0, K 2304, 40 rows 13.3 against 10.4 us), and a second CTA, up to 16 tokens with fp32
// scales and when a UE8M0 step has no prep blocks.
__host__ __device__ constexpr int bs_regs(int mp, bool wue, bool inl) { return wue ? (mp == 16 && inl ? 96 : 112) : mp == 16 ? 144 : 152; }
// Slabs an accumulator in tensor memory sums before the epilogue adds it up in fp32 registers.  The tensor cores
// truncate every addition, so a chain's error has a sign and grows with its length.  UE8M0, 2000 rows of 7168 x 8192,
// relative to 64-bit sums: all of K in one chain 4.9e-7 (scales spread over 2^24: 3.4e-6), four slabs 8.1e-8 (2.7e-7),
// two 9.2e-8 (1.8e-7), one 1.0e-7 (1.7e-7), at 124, 126, 131 and 160 us a step; up to 128 rows 2.2e-7 (1.7e-6), 6.8e-8
// (2.7e-7), 7.1e-8 (1.7e-7) and 7.6e-8 (1.4e-7).
__host__ __device__ constexpr int bs_chain(bool wue) { return wue ? 2 : 1; }
// Accumulators an epilogue thread reads at once: 64 registers' worth, UE8M0 (fewer registers a thread) 32.
__host__ __device__ constexpr int bs_read_batch(int mp, bool wue) {
    return (wue ? 32 : 64) / (mp * 4 / bs_epi_warps(mp)) > 0 ? (wue ? 32 : 64) / (mp * 4 / bs_epi_warps(mp)) : 1;
}
constexpr int kBsMaxAcc = 8;         // accumulator groups in tensor memory (a group = one stage's slabs)
constexpr int kBsMaxTokens = 128;    // activation rows one launch takes (16, 32, 64 or 128 MMA columns)
constexpr int kBsAtomBytes = 512;    // one scale atom: 128 rows x 4 K blocks
constexpr int kBsMmaRows = 128;      // M of the MMA; a tile of output rows holds at most as many

// Rows of a scale atom that exist in memory: the copy into tensor memory takes 32, those past the tokens'
// come from whatever follows and scale columns that are never read.  More than 128 tokens have two atoms.
__host__ __device__ constexpr int bs_atom_bytes(int m) { return m < 32 ? 16 * m : m <= 128 ? kBsAtomBytes : 2 * kBsAtomBytes; }

// The activation image of a step: the K slabs in the groups that the CTAs' stages take (half h of K owns slabs
// [h * ks / csize, (h + 1) * ks / csize), cut into groups of at most sl), a group being its chunks, then its atoms.
__host__ __device__ inline int bs_group(int slab, int ks, int csize, int sl, int &count) {  // first slab of the group, slabs in it
    const int half = ks / 2, lo = csize == 2 && slab >= half ? half : 0, hi = csize == 2 && slab < half ? half : ks;
    const int g0 = lo + (slab - lo) / sl * sl;
    count = sl < hi - g0 ? sl : hi - g0;
    return g0;
}

// ---------------------------------------------------------------- activation prep
struct ActPrepRank {
    const void *x;
    uint8_t *xq;  // see bs_group
    int64_t ldx;
};
struct ActPrepParams {
    int32_t m, k, x_dtype, ks, csize, sl;
    int32_t tokens, pad0;  // tokens per image: m, or (tile kernel) those of a tile, the tiles' images one after another
    ActPrepRank r[WS_MAX_WORLD];
};

// Thread = 16 values of one token at a time (two adjacent lanes share a 32-block); the K tail of the last
// slab is written as zeros.  Few threads per SM: beside 256 of them the main kernel's CTA found no registers
// and started late (measured at 40 rows: some CTAs 4.6 us after the predecessor's end instead of 1).
// AHEAD: the blocks are resident while the predecessor still runs, and ask for x then (not where x may be in host memory).
constexpr int kActPrepThreads = 128;
template <bool AHEAD>
__global__ void __launch_bounds__(kActPrepThreads, 12) act_prep_kernel(const __grid_constant__ ActPrepParams p) {
    // The step that follows may become resident at once (it streams weights until its own wait);
    // the activations come from earlier work on the stream.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const ActPrepRank &A = p.r[blockIdx.y];
    const int chunks = p.ks << 3, total = p.m * chunks, step = gridDim.x * kActPrepThreads;
    if constexpr (AHEAD)
        for (int c = blockIdx.x * kActPrepThreads + threadIdx.x; c < total; c += step) {
            const int tok = c / chunks, k = (c - tok * chunks) * 16;
            if (k < p.k) prefetch_act(A.x, p.x_dtype, (int64_t)tok * A.ldx + k);
        }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int U = 2;  // chunks whose loads are in flight together
    for (int c0 = blockIdx.x * kActPrepThreads + threadIdx.x; c0 - (int)(threadIdx.x & 31) < total; c0 += U * step) {  // whole warps
        float v[U][16];
        int tok[U], ch[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * step;
            tok[u] = c < total ? c / chunks : 0;
            ch[u] = c - tok[u] * chunks;
            const bool valid = c < total && ch[u] * 16 < p.k;
            load_act8(A.x, p.x_dtype, (int64_t)tok[u] * A.ldx + ch[u] * 16, valid, *reinterpret_cast<float(*)[8]>(v[u]));
            load_act8(A.x, p.x_dtype, (int64_t)tok[u] * A.ldx + ch[u] * 16 + 8, valid, *reinterpret_cast<float(*)[8]>(v[u] + 8));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int e;
            const uint4 q = act_quant16(v[u], e);
            if (c0 + u * step < total) {
                const int tile = tok[u] < p.tokens ? 0 : tok[u] / p.tokens, t = tok[u] - tile * p.tokens;
                const int m = min(p.tokens, p.m - tile * p.tokens), slab = ch[u] >> 3, atom = bs_atom_bytes(m);
                int count;
                const int g0 = bs_group(slab, p.ks, p.csize, p.sl, count);
                uint8_t *grp = A.xq + (int64_t)tile * p.ks * (p.tokens * 128 + bs_atom_bytes(p.tokens)) + (int64_t)g0 * (m * 128 + atom);
                *reinterpret_cast<uint4 *>(grp + ((int64_t)(ch[u] - g0 * 8) * m + t) * 16) = q;
                if ((ch[u] & 1) == 0)
                    grp[(int64_t)count * m * 128 + (slab - g0) * atom + (t >> 7) * kBsAtomBytes + (t & 31) * 16 + ((t >> 5) & 3) * 4 +
                        ((ch[u] >> 1) & 3)] = (uint8_t)min(max(e + 127, 0), 255);
            }
        }
    }
}

// ---------------------------------------------------------------- main kernel
struct alignas(64) BsParams {
    CUtensorMap tmap_w[WS_MAX_WORLD];  // weight shard [n][k bytes], box 128 bytes x tile_rows, 128B swizzle
    int32_t m, cols, n, k, ks, bn_shift, bk_shift;  // cols: N of the MMA, a multiple of 16 in [m, MP]
    int32_t world, mode, vocab, tmem_cols;  // tmem_cols: tensor-memory columns to allocate (512, or at most 256 when two CTAs share an SM)
    int32_t owner_reduce;              // all-reduce by owners: tile t is folded by rank t % world, which sends the sums back
    int32_t csize;                     // 1, or 2: CTA pairs (a cluster) share a tile, each streams half of K
    int32_t ahead;                     // the CTA asks for its activations ahead of the wait on the predecessor (INL)
    int32_t rx_behind;                 // CTA pairs: where the partner's sums arrive, see bs_smem_layout
    int32_t tile_rows, ntiles;         // output rows per tile (<= 128) and tiles of the shard
    int32_t slabs_per_stage, nstages;
    int32_t a_pitch, x_pitch;          // bytes one slab's weights (a multiple of 1024) / one stage's activations and atoms (of 128) occupy
    int32_t skb, nslot_max, nacc, gather_logits, x_dtype;
    uint64_t timeout_ns;
    SymLayout lay;
    Fp8RankArgs r[WS_MAX_WORLD];       // x is used when the kernel quantises itself (INL); the rest as in the decode kernels
    const uint8_t *xq[WS_MAX_WORLD];   // the prep kernel's activations and scale atoms
};

// Of a CTA pair, CTA r finishes the groups of four tokens 2 j + r: every epilogue thread then sends half of its columns and
// keeps half, in 16-byte words and without a test per column (each CTA half of the tokens in one run, a float at a time,
// took 4.6 us a tile at 96 rows and 1.0 at 19: 96 rows of K 8192 28.5 us a step, 25.5 now; 8 rows of K 1024 5.84, 5.28).
// Up to four rows are all CTA 0's, of twelve eight are: with peers its threads send and fold more words than equal halves
// would.  A last rank's step, the words of eight ranks at hand, takes the same time either way (3, 4, 12 rows 19.5, 19.5,
// 23.6 us); over NVLink it has not been timed.
__host__ __device__ constexpr int bs_rx_groups(int m) { return ((m + 3) / 4 + 1) / 2; }

struct BsSmem {
    int32_t a, x, wsf, sw, cand, rx, bars, misc, total;
};
__host__ __device__ inline BsSmem bs_smem_layout(int nstages, int slabs_per_stage, int a_pitch, int x_pitch, int nslot_max,
                                                 int skb, int mp, int rx_groups, bool rx_behind, bool wue, int x_resident) {
    BsSmem s{};
    const int nsl = nstages * slabs_per_stage;
    const int x_bytes = x_resident > 0 ? (x_resident + 127) / 128 * 128 : nstages * x_pitch;  // inline: all of this K half
    int o = 0;
    s.a = o;    o += nsl * a_pitch;
    s.x = o;    o += x_bytes;
    // an MMA reads 128 rows of its weight slab however many the tile holds, and up to 128 tokens and 32 atom
    // rows whatever m is: keep 16 KB readable behind the last slab and 2 KB behind the last activations.  What is there
    // goes into sums that nobody looks at: where room is short (bs_plan) a pair's exchange has its place there.
    const int behind = x_bytes + 2048 < kBsMmaRows * 128 ? kBsMmaRows * 128 - x_bytes : 2048, rx_bytes = rx_groups * kBsMmaRows * 16;
    s.rx = o;   o += rx_behind && rx_bytes > behind ? rx_bytes : behind;  // CTA pairs: the partner's sums of one tile for this CTA's tokens, [group of 4 tokens][row][4]
    s.wsf = o;  o += wue ? nsl * kBsAtomBytes : kBsAtomBytes;  // the weights' scale atoms (fp32 scales: one atom of 2^0)
    s.sw = o;   o += wue ? 0 : (int)align_up((int64_t)nslot_max * skb * 4, 16);
    s.cand = o; o += bs_epi_warps(mp) * mp * 8;          // lm_head: per epilogue warp and token (value, index)
    if (!rx_behind) { s.rx = o; o += rx_bytes; }
    s.bars = o; o += (2 * kMaxStages + kBsMaxAcc + 4) * 8;
    s.misc = o; o += 64;
    s.total = o;
    return s;
}

template <int MP, bool WUE, bool INL>
__device__ __forceinline__ BsSmem bs_layout(const BsParams &p) {
    return bs_smem_layout(p.nstages, p.slabs_per_stage, p.a_pitch, p.x_pitch, p.nslot_max, p.skb, MP, p.csize == 2 ? bs_rx_groups(p.m) : 0, p.rx_behind != 0, WUE,
                          INL ? (p.ks + p.csize - 1) / p.csize * (p.m * 128 + bs_atom_bytes(p.m)) : 0);
}

// ---- tcgen05 wrappers
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Shared-memory matrix descriptor, K-major: 128B swizzle with 8-row groups `sbo` bytes apart
// (operands), or no swizzle (scale atoms: 8-row x 16-byte core matrices `sbo` bytes apart).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t sbo, bool swizzle128) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);         // start address, 16-byte units
    if (swizzle128) d |= (uint64_t)1 << 16;           // leading byte offset: unused with 128B swizzle, K-major
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;      // stride between 8-row groups
    d |= (uint64_t)1 << 46;                           // descriptor version of sm_100
    if (swizzle128) d |= (uint64_t)2 << 61;           // SWIZZLE_128B
    return d;
}
// Instruction descriptor of the block-scaled MMA: E4M3 x E4M3, UE8M0 scales, M = 128, N = n;
// sfa / sfb pick the byte (K block of the slab) inside the scale operands' 32-bit columns.
__device__ __forceinline__ uint32_t bs_idesc(int n, int sfa, int sfb) {
    return ((uint32_t)sfb << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (8u << 24) |
           ((uint32_t)sfa << 29);
}
// D[tmem] (+)= A[smem] * B[smem] with per-32 scales from tensor memory.  The descriptors arrive as
// their 32-bit halves: the upper half is the same for every operand tile, the lower one advances by
// two (32 bytes) per K block, so the single issuing thread spends two adds per MMA on them.
__device__ __forceinline__ void umma_bs_ss(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t a_hi, uint32_t b_hi,
                                           uint32_t idesc, uint32_t tsfa, uint32_t tsfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %4};\n\t"
        "setp.ne.b32 p, %8, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], da, db, %5, [%6], [%7], p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(a_hi), "r"(b_hi), "r"(idesc), "r"(tsfa), "r"(tsfb), "r"(accumulate)
        : "memory");
}
// Halves of the 128B-swizzled K-major operand descriptor (see umma_desc): 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
constexpr uint32_t kUmmaDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);
// Upper half of the activation operand's descriptor: no swizzle, 8-token groups 128 bytes apart (the lower half
// carries the stride between 16-byte chunks of K).
constexpr uint32_t kUmmaDescHiX = (128u >> 4) | (1u << 14);
// One 512-byte scale atom (32 rows x 16 bytes) -> 4 columns of all 128 TMEM lanes.
__device__ __forceinline__ void tmem_cp_atom(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// N consecutive columns of this warp's 32 TMEM lanes -> registers; the wait is part of the same
// statement, so no use of the registers can be scheduled before the data has arrived.
#define WS_R4(a, i) "=r"(a[i]), "=r"(a[i + 1]), "=r"(a[i + 2]), "=r"(a[i + 3])
#define WS_R16(a, i) WS_R4(a, i), WS_R4(a, i + 4), WS_R4(a, i + 8), WS_R4(a, i + 12)
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[N]);
template <>
__device__ __forceinline__ void tmem_ld_cols<16>(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : WS_R16(r, 0) : "r"(taddr) : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_cols<32>(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : WS_R16(r, 0), WS_R16(r, 16) : "r"(taddr) : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_cols<64>(uint32_t taddr, uint32_t (&r)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
        "%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
        "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : WS_R16(r, 0), WS_R16(r, 16), WS_R16(r, 32), WS_R16(r, 48) : "r"(taddr) : "memory");
}
// The same N columns of B consecutive accumulators, `pitch` columns apart, under one wait.
template <int N, int B>
__device__ __forceinline__ void tmem_ld_batch(uint32_t taddr, uint32_t pitch, uint32_t (&r)[N * B]);
template <>
__device__ __forceinline__ void tmem_ld_batch<16, 4>(uint32_t t, uint32_t pitch, uint32_t (&r)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%65];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%66];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%67];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : WS_R16(r, 0), WS_R16(r, 16), WS_R16(r, 32), WS_R16(r, 48) : "r"(t), "r"(t + pitch), "r"(t + 2 * pitch), "r"(t + 3 * pitch) : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_batch<32, 2>(uint32_t t, uint32_t pitch, uint32_t (&r)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
        "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%65];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : WS_R16(r, 0), WS_R16(r, 16), WS_R16(r, 32), WS_R16(r, 48) : "r"(t), "r"(t + pitch) : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_batch<64, 1>(uint32_t t, uint32_t, uint32_t (&r)[64]) { tmem_ld_cols<64>(t, r); }
template <>
__device__ __forceinline__ void tmem_ld_batch<32, 1>(uint32_t t, uint32_t, uint32_t (&r)[32]) { tmem_ld_cols<32>(t, r); }
template <>
__device__ __forceinline__ void tmem_ld_batch<16, 2>(uint32_t t, uint32_t pitch, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : WS_R16(r, 0), WS_R16(r, 16) : "r"(t), "r"(t + pitch) : "memory");
}
#undef WS_R16
#undef WS_R4

// ---- distributed shared memory of a CTA pair
__device__ __forceinline__ uint32_t mapa_u32(uint32_t local_addr, uint32_t cta_rank) {  // the same address in CTA `cta_rank` of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(cta_rank));
    return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_f32x4(uint32_t addr, float a, float b, float c, float d) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t remote_bar) {  // releases this thread's earlier stores to the cluster
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
// Wait on an own barrier that the partner CTA arrives on; bounded like mbar_wait.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, uint32_t *status) {
    const uint64_t t0 = globaltimer_ns();
    uint32_t spins = 0;
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((++spins & 63u) == 0u) {
            if (*(volatile uint32_t *)status != 0u) return false;
            if (globaltimer_ns() - t0 > 2000000000ull) break;
        }
    }
    atomicCAS(status, 0u, kStatTimeoutTma | (uint32_t)(-WS_ERR_TIMEOUT));
    return false;
}

template <int THREADS>
__device__ __forceinline__ void bs_epi_bar_n() {  // the epilogue warps
    asm volatile("bar.sync 2, %0;" ::"n"(THREADS) : "memory");
}

// The sequence of stage items of one CTA.  The shard's rows are cut into tiles of tile_rows rows
// (at most 128, the M of the MMA; chosen so that the tiles deal out evenly) and CTA c takes tiles
// [c * T / ncta, (c + 1) * T / ncta) whole, so every output row is a complete dot product inside one
// CTA and nothing is combined across CTAs.  An item is up to SL consecutive K slabs of one tile.
// With CTA pairs (csize = 2) the tiles are dealt out to the pairs and each CTA of a pair walks one
// half of every tile's K slabs; the second CTA hands its sums to the first through the pair's
// distributed shared memory (see the epilogue).
struct BsWalk {
    int t, t1, s, K0, K1, SL;  // tiles [t, t1), slabs [K0, K1) of each
    __device__ __forceinline__ BsWalk(int ntiles, int part, int nparts, int k0, int k1, int sl) : s(k0), K0(k0), K1(k1), SL(sl) {
        t = (int)((int64_t)ntiles * part / nparts);
        t1 = (int)((int64_t)ntiles * (part + 1) / nparts);
        if (k1 <= k0) t1 = t;
    }
    // next item: tile, first slab, slab count; false when the CTA's tiles are used up
    __device__ __forceinline__ bool next(int &tile, int &s0, int &nsl) {
        if (t >= t1) return false;
        tile = t;
        s0 = s;
        nsl = min(SL, K1 - s);
        s += nsl;
        if (s == K1) {
            s = K0;
            ++t;
        }
        return true;
    }
};

// UE8M0 weight scales of a shard as scale-operand words: the four exponents of a row's 128-wide K slab (2^0 past the
// end of K).  32-wide blocks on word boundaries are one load; collected byte by byte with an address each, a warp's
// instructions took longer than the slab's MMAs.
struct Ue8m0Scales {
    const uint8_t *base;
    int64_t ld, k0;
    int k, bk_shift;
    bool words;
    __device__ __forceinline__ Ue8m0Scales(const void *scales, int64_t ld_, int64_t k0_, int k_, int bk_shift_)
        : base(static_cast<const uint8_t *>(scales)), ld(ld_), k0(k0_), k(k_), bk_shift(bk_shift_) {
        words = bk_shift == 5 && (k0 & 127) == 0 && (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(base) & 3) == 0;
        if (words) base += k0 >> 5;
    }
    __device__ __forceinline__ const uint8_t *row(int64_t scale_row) const { return base + scale_row * ld; }
    __device__ __forceinline__ uint32_t slab(const uint8_t *row, int s) const {
        const int left = k - s * 128;  // a multiple of 32
        uint32_t v = 0x7F7F7F7Fu;
        if (words) {
            v = __ldg(reinterpret_cast<const uint32_t *>(row) + s);
            if (left < 128) v = (v & ((1u << (left >> 2)) - 1u)) | (0x7F7F7F7Fu << (left >> 2));
        } else {
#pragma unroll 1
            for (int q = 0; q < 4 && q * 32 < left; ++q)
                v = (v & ~(0xFFu << (8 * q))) | (uint32_t)__ldg(row + ((k0 + s * 128 + q * 32) >> bk_shift)) << (8 * q);
        }
        return v;
    }
};

// Floats in an order that unsigned comparison keeps; everything that is not above -inf is 0.
__device__ __forceinline__ uint32_t order_key(float v) {
    if (!(v > -INFINITY)) return 0u;
    const uint32_t b = __float_as_uint(v + 0.0f);  // -0 and +0 are equal
    return b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}
__device__ __forceinline__ float order_value(uint32_t key) { return __uint_as_float(key ^ ((key >> 31) ? 0x80000000u : 0xFFFFFFFFu)); }

// Sums, in rank order, of `count` (<= T) tokens' words of one output row: those of all ranks (R = WS_MAX_WORLD; src is
// rank 0's) or one rank's (R = 1).  All of them are requested before the first is looked at, one memory round trip
// instead of one per rank (three rows on eight ranks: 29 of a 50 us step), and requested again while one is missing:
// waiting for each missing word in turn took a round trip per word (40 rows on eight ranks 198 us a step, 72 now; two
// tokens at a time 87).  A rank that stays away is left to wait_word, which
// gives up and records it; false then: the sums are void.
// Word i is that of token (i & 3) + (i >> 2) * gap of the T; those at or past `count` are not there.
constexpr int kFoldTokens = 4, kFoldTries = 256;
template <int T, int R>
__device__ __forceinline__ bool fold_words(const BsParams &p, const RankCtx &X, const uint64_t *src, size_t astride, uint32_t seq, int count, int gap,
                                           float (&sum)[T]) {
    auto token = [&](int i) { return (i & 3) + (i >> 2) * gap; };
    const int ranks = R == 1 ? 1 : p.world;
    bool here = false;
#pragma unroll 1
    for (int tries = 0; tries < kFoldTries && !here; ++tries) {
        if ((tries & 15) == 15 && *(volatile uint32_t *)X.status != 0u) break;  // the step has failed already
        uint64_t w[R][T];
        const uint64_t *at = src;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
            if (R == 1 || rr < ranks) {
#pragma unroll
                for (int i = 0; i < T; ++i) w[rr][i] = ld_word_sys(at + (int64_t)(token(i) < count ? token(i) : 0) * p.n);
            }
            at += astride;
        }
        here = true;
#pragma unroll
        for (int rr = 0; rr < R; ++rr)
            if (R == 1 || rr < ranks) {
#pragma unroll
                for (int i = 0; i < T; ++i) {
                    here = here && (uint32_t)(w[rr][i] >> 32) == seq;
                    const float v = __uint_as_float((uint32_t)w[rr][i]);
                    sum[i] = rr == 0 ? v : sum[i] + v;
                }
            }
    }
    if (here) return true;
#pragma unroll
    for (int i = 0; i < T; ++i) {
        sum[i] = 0.0f;
        if (token(i) < count)
#pragma unroll 1
            for (int rr = 0; rr < ranks; ++rr) {
                const float v = wait_word(src + rr * astride + (int64_t)token(i) * p.n, seq, p.timeout_ns, X.status, kStatTimeoutPeerA);
                sum[i] = rr == 0 ? v : sum[i] + v;
            }
    }
    return *(volatile uint32_t *)X.status == 0u;
}

// The exchange behind a CTA's finished tiles: fold its rows, in rank order, as the ranks' words arrive.  Thread
// `et` of the epilogue (32 * ew of them) takes row et % 128 of each tile and the tokens whose columns it held.  A
// function of its own, called when nothing else is left to do: inside the epilogue what it holds in registers was
// taken from the main loops (three rows of K 8192 on one rank 16.0 us instead of 15.0).
static __device__ __noinline__ void bs_fold(const BsParams &p, int ew, int cp) {
    const int vr = blockIdx.y, pair = p.csize == 2 ? 1 : 0;
    const Fp8RankArgs &A = p.r[vr];
    const RankCtx &X = A.ctx;
    const uint32_t seq = step_begin(X), bank = seq & 1u;
    const int TR = p.tile_rows, part = blockIdx.x >> pair, nparts = gridDim.x >> pair;
    const int t_lo = (int)((int64_t)p.ntiles * part / nparts), t_hi = (int)((int64_t)p.ntiles * (part + 1) / nparts) - 1;
    const int warp = (int)(threadIdx.x >> 5), rc = (warp & 3) * 32 + (int)(threadIdx.x & 31), col0 = ((warp - 2) >> 2) * cp;
    // this thread's tokens: all of its columns', or, of a pair, every other group of four
    const int tbeg = col0 + (pair ? 4 * (int)(blockIdx.x & 1) : 0), tend = min(p.m, col0 + cp), gap = pair ? 8 : 4;
    if (warp < 2 || warp >= 2 + ew) return;
    const size_t astride = (size_t)p.lay.max_m * p.lay.max_n;
    const uint64_t *slots = reinterpret_cast<const uint64_t *>(X.sym[X.rank] + p.lay.slota_off) + (size_t)bank * p.world * astride;
    // Fold by owners (owner_reduce): the sums of tile t are formed on rank t % world only (in rank order, as
    // everywhere) and travel back in that rank's own slot at every peer, so all ranks end up with the same bits and
    // each partial sum crosses the links once instead of world - 1 times.  A rank folds its own tiles before it
    // collects the others': the owners do not wait for one another.
    for (int pass = p.owner_reduce ? 0 : 1; pass < 2; ++pass)
        for (int t = t_lo; t <= t_hi; ++t) {
            const int row = t * TR + rc;
            if (rc >= TR || row >= p.n) continue;
            const int owner = p.owner_reduce ? t % p.world : X.rank;
            if (p.owner_reduce && (owner == X.rank) != (pass == 0)) continue;
            const uint64_t *src = slots + (size_t)tbeg * p.n + row;
            float *out = A.out + (size_t)tbeg * p.n + row;
            if (owner != X.rank) {
                for (int tok = tbeg; tok < tend; tok += 2 * gap, src += 2 * gap * (int64_t)p.n, out += 2 * gap * (int64_t)p.n) {
                    float sum[8];
                    fold_words<8, 1>(p, X, src + owner * astride, astride, seq, tend - tok, gap, sum);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int o = (i & 3) + (i >> 2) * gap;
                        if (tok + o < tend) out[(int64_t)o * p.n] = sum[i];
                    }
                }
                continue;
            }
            for (int tok = tbeg; tok < tend; tok += gap, src += gap * (int64_t)p.n, out += gap * (int64_t)p.n) {
                float sum[kFoldTokens];
                const bool valid = fold_words<kFoldTokens, WS_MAX_WORLD>(p, X, src, astride, seq, tend - tok, gap, sum);
#pragma unroll
                for (int i = 0; i < kFoldTokens; ++i)
                    if (tok + i < tend) out[(int64_t)i * p.n] = sum[i];
                if (p.owner_reduce && valid)  // (the others time out, too, rather than take what was folded without a rank)
                    for (int pr = 0; pr < p.world; ++pr) {
                        if (pr == X.rank) continue;
                        uint64_t *dst = reinterpret_cast<uint64_t *>(X.sym[pr] + p.lay.slota_off) +
                                        ((size_t)bank * p.world + X.rank) * astride + (size_t)tok * p.n + row;
#pragma unroll
                        for (int i = 0; i < kFoldTokens; ++i)
                            if (tok + i < tend) st_word_sys(dst + (int64_t)i * p.n, seq, sum[i]);
                    }
            }
        }
}

// What follows a CTA's finished tiles in an lm_head step, by its epilogue warps.  The argmax: the CTAs of a rank leave
// their candidates in the rank's own table; the CTA that arrives last merges them into ONE (value, lowest index) per
// token, sends it to every peer and merges the ranks' candidates: one 64-bit store and one flag per peer and step instead
// of one per CTA.  Then the gathered logits.  A function of its own, which finds its shared memory itself, for the same
// reason as bs_fold: inside the epilogue it cost the main loops of 64 rows their registers (an all-reduce step of 40 rows
// 21.3 us instead of 19.8; 64 rows of logits over 62944 x 4352 77.7 instead of 64.2).
template <int MP, bool WUE, bool INL>
static __device__ __noinline__ void bs_lm_head(const BsParams &p) {
    constexpr int EW = bs_epi_warps(MP), ET = EW * 32, CP = MP * 4 / EW;
    if (threadIdx.x < 64 || threadIdx.x >= 64 + ET) return;
    extern __shared__ uint8_t smem_raw[];
    const BsSmem S = bs_layout<MP, WUE, INL>(p);
    uint8_t *smem = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw));
    const float *cv_s = reinterpret_cast<const float *>(smem + S.cand);
    const uint32_t *ci_s = reinterpret_cast<const uint32_t *>(smem + S.cand) + EW * MP;
    volatile uint32_t *last_s = reinterpret_cast<uint32_t *>(smem + S.misc) + 4;
    auto bs_epi_bar = [] { bs_epi_bar_n<ET>(); };
    const Fp8RankArgs &A = p.r[blockIdx.y];
    const RankCtx &X = A.ctx;
    const int et = (int)threadIdx.x - 64, ew = et >> 5, lane = et & 31, cta = blockIdx.x, ncta = gridDim.x;
    const uint32_t seq = step_begin(X), bank = seq & 1u;
    const int nflag = kMaxCtas + kMaxShared;
    const uint32_t *myflags = reinterpret_cast<const uint32_t *>(X.sym[X.rank] + p.lay.flags_off) + (size_t)bank * p.world * nflag;
    bs_epi_bar();
    auto pairs_of = [&](int r) { return reinterpret_cast<uint64_t *>(X.sym[r] + p.lay.pairs_off) + (size_t)bank * p.world * kMaxCtas * p.lay.max_m; };
    uint64_t *table = pairs_of(X.rank) + (size_t)X.rank * p.lay.max_m * kMaxCtas;  // [token][CTA]
    if (et < p.m) {  // token et: the four warps (one per lane quarter) that hold its column
        const int w0 = (et / CP) * 4;
        float bv = cv_s[w0 * MP + et];
        uint32_t bi = ci_s[w0 * MP + et];
        for (int w = w0 + 1; w < w0 + 4; ++w)
            if (cand_better(cv_s[w * MP + et], ci_s[w * MP + et], bv, bi)) { bv = cv_s[w * MP + et]; bi = ci_s[w * MP + et]; }
        table[(size_t)et * kMaxCtas + cta] = ((uint64_t)__float_as_uint(bv) << 32) | bi;
    }
    bs_epi_bar();
    if (et == 0) {
        __threadfence();
        const bool last = atomicAdd(X.counters, 1u) + 1u == (uint32_t)ncta;
        if (last) {
            X.counters[0] = 0u;  // ready for the next step
            __threadfence();
        }
        *last_s = last ? 1u : 0u;
    }
    bs_epi_bar();
    if (*last_s) {
        constexpr int kRankSlot = kMaxCtas - 1;  // a token's slot for the rank's merged candidate (a rank runs fewer CTAs than that)
        // Best of `count` (at most kMaxCtas) entries of the tokens t, t + EW, ...: a warp requests all entries of four
        // tokens before it looks at the first (one by one, the merge of 15 tokens was 10 us of a 30 us step).
        auto merge = [&](int count, auto entry, auto done) {
            constexpr int U = 4, J = kMaxCtas / 32;
            static_assert(kMaxCtas % 32 == 0, "every entry has a lane");
            for (int t0 = ew; t0 < p.m; t0 += U * EW) {
                uint64_t pr[U][J];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int j = 0; j < J; ++j)
                        if (t0 + u * EW < p.m && j * 32 + lane < count) pr[u][j] = ld_volatile_u64(entry(t0 + u * EW, j * 32 + lane));
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (t0 + u * EW >= p.m) break;
                    float bv = -INFINITY;
                    uint32_t bi = 0xFFFFFFFFu;
#pragma unroll
                    for (int j = 0; j < J; ++j) {
                        const float v = __uint_as_float((uint32_t)(pr[u][j] >> 32));
                        if (j * 32 + lane < count && cand_better(v, (uint32_t)pr[u][j], bv, bi)) { bv = v; bi = (uint32_t)pr[u][j]; }
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                        const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                        if (cand_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
                    }
                    done(t0 + u * EW, bv, bi);
                }
            }
        };
        auto answer = [&](int t, float, uint32_t bi) {
            if (lane == 0 && A.argmax != nullptr) A.argmax[t] = bi == 0xFFFFFFFFu ? 0u : bi;
        };
        auto own = [&](int t, int i) { return table + (size_t)t * kMaxCtas + i; };
        if (p.world == 1) {
            merge(ncta, own, answer);
        } else {
            merge(ncta, own, [&](int t, float bv, uint32_t bi) {
                if (lane < p.world)
                    pairs_of(lane)[((size_t)X.rank * p.lay.max_m + t) * kMaxCtas + kRankSlot] = ((uint64_t)__float_as_uint(bv) << 32) | bi;
            });
            bs_epi_bar();  // the st.release.sys below is cumulative over the stores this barrier ordered
            if (et < p.world) {
                uint32_t *f = reinterpret_cast<uint32_t *>(X.sym[et] + p.lay.flags_off) + ((size_t)bank * p.world + X.rank) * nflag;
                st_release_sys(f + kMaxCtas + 1, seq);
                wait_flag(myflags + (size_t)et * nflag + kMaxCtas + 1, seq, p.timeout_ns, X.status, kStatTimeoutGather);
            }
            bs_epi_bar();
            merge(p.world, [&](int t, int r) { return pairs_of(X.rank) + ((size_t)r * p.lay.max_m + t) * kMaxCtas + kRankSlot; }, answer);
        }
    }
    if (p.gather_logits && p.world > 1) {
        // every CTA's rows are in every rank's gather buffer once its flag is there (the barriers above
        // order the stores before this release); each CTA then copies a share of the vocabulary out
        if (et < p.world) {
            uint32_t *f = reinterpret_cast<uint32_t *>(X.sym[et] + p.lay.flags_off) + ((size_t)bank * p.world + X.rank) * nflag;
            st_release_sys(f + cta, seq);
        }
        if (A.logits != nullptr) {
            for (int i = et; i < p.world * ncta; i += ET)
                wait_flag(myflags + (size_t)(i / ncta) * nflag + (i % ncta), seq, p.timeout_ns, X.status, kStatTimeoutGather);
            bs_epi_bar();
            const float *gl = reinterpret_cast<const float *>(X.sym[X.rank] + p.lay.gather_off) +
                              (size_t)bank * p.lay.max_m * (size_t)p.lay.max_vocab;
            const int64_t per = ((int64_t)p.vocab + ncta - 1) / ncta;
            const int64_t v0 = (int64_t)cta * per, v1 = min((int64_t)p.vocab, v0 + per);
            for (int tok = 0; tok < p.m; ++tok)
                for (int64_t v = v0 + et; v < v1; v += ET)
                    A.logits[(size_t)tok * p.vocab + v] = __ldcg(gl + (size_t)tok * p.lay.max_vocab + v);
        }
    }
}

template <int MP, bool WUE, bool INL>
__global__ void __launch_bounds__(bs_threads(MP, WUE)) __maxnreg__(bs_regs(MP, WUE, INL)) fp8_bs_kernel(const __grid_constant__ BsParams p) {
    constexpr int EW = bs_epi_warps(MP), ET = EW * 32;  // epilogue warps / threads
    constexpr int CP = MP * 4 / EW;                      // token columns one epilogue thread holds
    auto bs_epi_bar = [] { bs_epi_bar_n<ET>(); };
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);

    const int vr = blockIdx.y, cta = blockIdx.x, ncta = gridDim.x;
    const Fp8RankArgs &A = p.r[vr];
    const RankCtx &X = A.ctx;
    const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;

    const int KS = p.ks;                                    // slabs per tile
    // CTA pairs: which half of K is this CTA's, and which pair of how many it belongs to
    uint32_t crank = 0;
    if (p.csize == 2) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    const int part = p.csize == 2 ? cta >> 1 : cta, nparts = p.csize == 2 ? ncta >> 1 : ncta;
    const int k_lo = (int)crank * KS / p.csize, k_hi = ((int)crank + 1) * KS / p.csize;
    constexpr int CH = bs_chain(WUE);
    const int SL = p.slabs_per_stage, NS = p.nstages, NB = p.nacc, AS = (SL + CH - 1) / CH;  // AS accumulators per stage
    const int ntiles = p.ntiles, TR = p.tile_rows;

    const BsSmem S = bs_layout<MP, WUE, INL>(p);
    float *sw_s = reinterpret_cast<float *>(smem + S.sw);
    uint32_t *misc_s = reinterpret_cast<uint32_t *>(smem + S.misc);
    const uint32_t a0 = smem_u32(smem + S.a), x0 = smem_u32(smem + S.x), wsf0 = smem_u32(smem + S.wsf);
    // full[s]: the stage's bytes landed (UE8M0: and the auxiliary warps have written its weight scales).
    // done[s]: every MMA that reads the stage has completed (ONE tcgen05.commit per stage: a commit stalls
    // the issuing thread for ~160 ns, so it is not spent per slab).  A stage's slabs accumulate into the AS
    // buffers of accumulator group g = item mod NB, done[s] also tells the epilogue that they are ready,
    // accempty[g] that the group has been read back.
    const uint32_t full0 = smem_u32(smem + S.bars), done0 = full0 + kMaxStages * 8;
    const uint32_t accempty0 = done0 + kMaxStages * 8;
    const uint32_t rxfull = accempty0 + kBsMaxAcc * 8, rxempty = rxfull + 8, xready = rxempty + 8;  // CTA pairs: the partner's sums of a tile have arrived / been read

    // Weights are static: the first ring's worth is on its way before the CTA has set itself up (barriers,
    // tensor memory and the pair's meeting take ~1.3 us, in which HBM would idle), let alone before the wait on
    // the prep kernel.
    const uint32_t x_slab = (uint32_t)(p.m * 128 + bs_atom_bytes(p.m));
    auto issue_w = [&](int s, int tile, int s0, int nsl) {
        mbar_arrive_expect_tx(full0 + s * 8, (uint32_t)nsl * ((uint32_t)TR * 128u + (INL ? 0u : x_slab)));
        for (int j = 0; j < nsl; ++j)
            tma_load_2d(a0 + (s * SL + j) * p.a_pitch, &p.tmap_w[vr], (s0 + j) * 128, tile * TR, full0 + s * 8);
    };
    if (warp == 0) {
        if (elect_one()) {
            for (int s = 0; s < NS; ++s) {
                mbar_init(full0 + s * 8, WUE ? 1 + kBsAuxWarps : 1);
                mbar_init(done0 + s * 8, 1);
            }
            for (int b = 0; b < kBsMaxAcc; ++b) mbar_init(accempty0 + b * 8, EW);  // one arrival per epilogue warp
            mbar_init(rxfull, EW);   // every epilogue warp of the partner arrives after its stores
            mbar_init(rxempty, EW);
            mbar_init(xready, EW);   // inline: the activations are in shared memory
            mbar_fence_init();
            int tile, s0, nsl;
            BsWalk w(ntiles, part, nparts, k_lo, k_hi, SL);
            for (int item = 0; item < NS && w.next(tile, s0, nsl); ++item) issue_w(item, tile, s0, nsl);
        }
        __syncwarp();
    }
    if constexpr (INL) {
        if (p.ahead && warp >= 2 && warp < 2 + EW)
            for (int c = tid - 64, chunks = (k_hi - k_lo) * 8; c < p.m * chunks; c += ET) {
                const int tok = c / chunks, k = k_lo * 128 + (c - tok * chunks) * 16;
                if (k < p.k) prefetch_act(A.x, p.x_dtype, (int64_t)tok * A.ldx + k);
            }
    }
    if (warp == 1) {  // tensor memory: allocated and freed by the same warp
        tmem_alloc(smem_u32(misc_s), (uint32_t)p.tmem_cols);
        tmem_relinquish();
    }
    if (!WUE && warp >= 2 && warp < 6) {  // the weight operand's scale atom: 2^0 everywhere (128 threads x 4 bytes)
        reinterpret_cast<uint32_t *>(smem + S.wsf)[tid - 64] = 0x7F7F7F7Fu;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (p.csize == 2) {  // the partner's barriers are initialised before anything is sent to them
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(misc_s);
    // tensor-memory columns: NB groups x AS accumulator buffers of MP columns.  Then, fp32 weight scales: 4
    // activation-scale columns (one scale atom) per buffer, the 4 weight-scale columns.  UE8M0: for two stages
    // and SL slabs each 4 activation- and 4 weight-scale columns.
    const uint32_t t_sf0 = tmem_base + (uint32_t)(NB * AS * MP);
    const uint32_t t_sfa = t_sf0 + (uint32_t)(NB * SL * 4);  // fp32 weight scales only
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == 0) {
        // ------------------------------------------------------------ producer (one thread)
        if (elect_one()) {
            int tile, s0, nsl;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            BsWalk w(ntiles, part, nparts, k_lo, k_hi, SL);
            RingPos st;
            for (int item = 0; w.next(tile, s0, nsl); ++item, st.next(NS)) {
                const int s = st.s;
                if (item >= NS) {
                    if (!mbar_wait(done0 + s * 8, st.ph ^ 1u, X.status)) break;
                    issue_w(s, tile, s0, nsl);
                }
                if (!INL) bulk_load(x0 + s * p.x_pitch, p.xq[vr] + (size_t)s0 * x_slab, (uint32_t)nsl * x_slab, full0 + s * 8);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issue (one thread)
        // A second issuing thread (stage items taken in turn, so that one thread's waits and commit hide
        // behind the other's MMAs) was ~7% faster on one-row steps, but a launch that streamed a
        // [129280, 7168] shard partly out of L2 (weights written just before) then ended in "unspecified
        // launch failure" in most attempts, in a different CTA and stage item each time, and never with
        // one thread; the barrier hand-offs are the same either way, so the cause is not known.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (elect_one()) {
            if (!WUE) tmem_cp_atom(t_sfa, umma_desc(wsf0, 128, false));
            // The tensor pipe runs on for ~200 clocks after the last MMA it was given, so what this thread does
            // between two stages has to stay below that: everything is an add away, the waits are on barriers
            // whose phase is usually complete.
            uint32_t id[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) id[q] = bs_idesc(p.cols, WUE ? q : 0, q);
            uint32_t *const status = X.status;
            const uint32_t m16 = (uint32_t)p.m;  // 16-byte units: one chunk of all tokens
            const uint32_t a_step = (uint32_t)p.a_pitch >> 4, x_step = 8u * m16, x_kb = 2u * m16, xsf_step = (uint32_t)bs_atom_bytes(p.m) >> 4;
            constexpr uint32_t kSfStep = (uint32_t)kBsAtomBytes >> 4;
            // of the current stage: barrier, operand descriptors (low halves), scale atoms; and of ring start
            const uint32_t a_stage = (uint32_t)SL * a_step, x_stage = (uint32_t)p.x_pitch >> 4;
            const uint32_t a_lo0 = umma_desc_lo(a0), x_lo0 = ((x0 & 0x3FFFFu) >> 4) | (m16 << 16);
            const uint64_t xsf0 = umma_desc(x0, 128, false), wsf_desc0 = umma_desc(wsf0, 128, false);
            uint32_t full = full0, done = done0, a_lo = a_lo0, x_lo = x_lo0, x_off = 0, w_off = 0, ph = 0;
            const uint32_t full_end = full0 + NS * 8;
            // accumulator ring
            uint32_t accempty = accempty0, t_acc = tmem_base, t_sf = t_sf0, acc_ph = 1;
            const uint32_t acc_end = accempty0 + NB * 8;
            constexpr bool inl = INL;
            uint32_t sf_off = 0;
            // one stage: straight-line code per slab count (a rolled loop costs twice the time)
            auto issue = [&](auto count) {
                constexpr int C = decltype(count)::value;
                const uint64_t xsf = xsf0 + (uint64_t)(inl ? sf_off : x_off + (uint32_t)C * x_step), wsf = wsf_desc0 + (uint64_t)w_off;
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    const uint32_t a = a_lo + (uint32_t)j * a_step, b = x_lo + (uint32_t)j * x_step;
                    const uint32_t d = t_acc + (uint32_t)(j / CH * MP);
                    const uint32_t sx = t_sf + (uint32_t)(j * (WUE ? 8 : 4)), sw = WUE ? sx + 4 : t_sfa;
                    tmem_cp_atom(sx, xsf + (uint64_t)((uint32_t)j * xsf_step));
                    if (WUE) tmem_cp_atom(sw, wsf + (uint64_t)(j * kSfStep));
                    umma_bs_ss(d, a, b, kUmmaDescHiSw128, kUmmaDescHiX, id[0], sw, sx, j % CH ? 1u : 0u);
                    umma_bs_ss(d, a + 2, b + x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id[1], sw, sx, 1u);
                    umma_bs_ss(d, a + 4, b + 2 * x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id[2], sw, sx, 1u);
                    umma_bs_ss(d, a + 6, b + 3 * x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id[3], sw, sx, 1u);
                }
            };
            const int my_tiles = (int)((int64_t)ntiles * (part + 1) / nparts) - (int)((int64_t)ntiles * part / nparts), kcta = k_hi - k_lo;
            const uint32_t sf_off0 = (uint32_t)kcta * x_step;  // inline: the atoms follow all of the K half's activations
            bool ok = !INL || mbar_wait(xready, 0, status);
            uint32_t odd = 0;  // UE8M0: which of the two sets of scale columns
            for (int t = kcta > 0 ? my_tiles : 0; t > 0 && ok; --t) {
                if (inl) { x_lo = x_lo0; sf_off = sf_off0; }
                for (int left = kcta; left > 0; left -= SL) {
                    if (!mbar_wait(accempty, acc_ph, status)) { ok = false; break; }
                    if (!mbar_wait(full, ph, status)) { ok = false; break; }
                    tc_fence_after();
                    if (left >= 4 && SL == 4) issue(std::integral_constant<int, 4>{});
                    else if (left >= 3 && SL >= 3) issue(std::integral_constant<int, 3>{});
                    else if (left >= 2 && SL >= 2) issue(std::integral_constant<int, 2>{});
                    else issue(std::integral_constant<int, 1>{});
                    umma_commit(done);  // the stage may be refilled and its accumulators read
                    // next stage
                    full += 8; done += 8; a_lo += a_stage; x_off += x_stage;
                    x_lo += inl ? (uint32_t)SL * x_step : x_stage;
                    sf_off += (uint32_t)SL * xsf_step;
                    if (WUE) w_off += (uint32_t)SL * kSfStep;
                    if (full == full_end) {
                        full = full0; done = done0; a_lo = a_lo0; x_off = 0; w_off = 0;
                        if (!inl) x_lo = x_lo0;
                        ph ^= 1u;
                    }
                    // next accumulator group
                    accempty += 8;
                    t_acc += (uint32_t)(AS * MP);
                    if (!WUE) t_sf += (uint32_t)(SL * 4);
                    if (accempty == acc_end) {
                        accempty = accempty0; t_acc = tmem_base;
                        if (!WUE) t_sf = t_sf0;
                        acc_ph ^= 1u;
                    }
                    if (WUE) {
                        odd ^= 1u;
                        t_sf = t_sf0 + odd * (uint32_t)(SL * 8);
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp >= 2 + EW) {
        // ------------------------------------------------------------ auxiliary warps (UE8M0 weight scales)
        // The scale bytes of the tile's rows (thread = row) become the stage's scale atoms; static, so they do not
        // wait for the predecessor.  Three items' words are in flight.
        if constexpr (WUE) {
            const int r = tid - 64 - ET;
            const Ue8m0Scales sc(A.scales, A.scale_ld, A.k0, p.k, p.bk_shift);
            BsWalk w(ntiles, part, nparts, k_lo, k_hi, SL);
            RingPos st;
            int item = 0;
            uint32_t at = smem_u32(smem + S.wsf) + (uint32_t)((r & 31) * 16 + (r >> 5) * 4);
            const uint32_t at_step = (uint32_t)(SL * kBsAtomBytes), at_end = at + NS * at_step;
            auto load = [&](uint32_t (&b)[4]) {  // the next item's words; returns its slab count, 0 behind the last
                int tile, s0, nsl;
                if (!w.next(tile, s0, nsl)) return 0;
                const uint8_t *row = sc.row((A.row0 + min(tile * TR + r, p.n - 1)) >> p.bn_shift);
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = sc.slab(row, min(s0 + j, k_hi - 1));
                return nsl;
            };
            auto put = [&](const uint32_t (&b)[4], int nsl) {
                bool ok = nsl > 0;
                if (item == NS) wait_predecessor();
                if (ok && item >= NS) ok = mbar_wait(done0 + st.s * 8, st.ph ^ 1u, X.status);
                if (!__all_sync(0xffffffffu, ok)) return false;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < nsl) asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + j * kBsAtomBytes), "r"(b[j]) : "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + st.s * 8);
                ++item;
                st.next(NS);
                at += at_step;
                if (at == at_end) at -= NS * at_step;
                return true;
            };
            uint32_t b0[4], b1[4], b2[4];
            int n0 = load(b0), n1 = load(b1), n2 = load(b2);
            for (;;) {
                if (!put(b0, n0)) break;
                n0 = load(b0);
                if (!put(b1, n1)) break;
                n1 = load(b1);
                if (!put(b2, n2)) break;
                n2 = load(b2);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue warps
        const int et = tid - 64;                     // 0..ET-1
        const int ew = warp - 2;                     // 0..EW-1
        const int quad = warp & 3;                   // TMEM lanes this warp may read: its index modulo 4
        const int rc = quad * 32 + lane;             // row inside the tile = TMEM lane
        const int col0 = (ew >> 2) * CP;             // first token column of this thread
        const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
        const int t_lo = (int)((int64_t)ntiles * part / nparts), t_hi = (int)((int64_t)ntiles * (part + 1) / nparts) - 1;  // this CTA's tiles
        const int64_t kcol0 = A.k0 >> p.bk_shift;
        const int64_t srow_lo = (A.row0 + t_lo * TR) >> p.bn_shift;
        if constexpr (!WUE) {
            // weight scales of the rows this CTA touches as fp32: sw_s[slot][column].  They are static, so
            // they are fetched before the wait on the predecessor.
            const int row_lo = t_lo * TR, row_hi = min(p.n, (t_hi + 1) * TR);
            const int nslot = row_hi > row_lo ? (int)(((A.row0 + row_hi - 1) >> p.bn_shift) - srow_lo + 1) : 0;
            const int ncols = (int)(((A.k0 + p.k - 1) >> p.bk_shift) - kcol0 + 1);
            for (int i = et; i < nslot * ncols; i += ET) {
                const int sl = i / ncols, c = i - sl * ncols;
                sw_s[sl * p.skb + c] = __ldg(static_cast<const float *>(A.scales) + (srow_lo + sl) * A.scale_ld + kcol0 + c);
            }
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if constexpr (INL) {  // few enough values: this CTA's K half of the activations, straight into shared memory
            const int chunks = (k_hi - k_lo) * 8, total = p.m * chunks, atom = bs_atom_bytes(p.m);
            uint8_t *xs = smem + S.x, *atoms = xs + (size_t)total * 16;
            constexpr int U = 2;  // chunks whose loads are in flight together
            for (int c0 = et; c0 - lane < total; c0 += U * ET) {  // whole warps
                float v[U][16];
                int tok[U], ch[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int c = c0 + u * ET;
                    tok[u] = c < total ? c / chunks : 0;
                    ch[u] = c - tok[u] * chunks;
                    const int kk = k_lo * 128 + ch[u] * 16;
                    const bool valid = c < total && kk < p.k;
                    load_act8(A.x, p.x_dtype, (int64_t)tok[u] * A.ldx + kk, valid, *reinterpret_cast<float(*)[8]>(v[u]));
                    load_act8(A.x, p.x_dtype, (int64_t)tok[u] * A.ldx + kk + 8, valid, *reinterpret_cast<float(*)[8]>(v[u] + 8));
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    int e;
                    const uint4 q = act_quant16(v[u], e);
                    if (c0 + u * ET < total) {
                        *reinterpret_cast<uint4 *>(xs + ((size_t)ch[u] * p.m + tok[u]) * 16) = q;
                        if ((ch[u] & 1) == 0)
                            atoms[(size_t)(ch[u] >> 3) * atom + (tok[u] & 31) * 16 + (tok[u] >> 5) * 4 + ((ch[u] >> 1) & 3)] =
                                (uint8_t)min(max(e + 127, 0), 255);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(xready);
        }
        const uint32_t seq = step_begin(X);
        const uint32_t bank = seq & 1u;
        bs_epi_bar();
        const int kofs = (int)(A.k0 - kcol0 * ((int64_t)1 << p.bk_shift));
        const bool solo = p.mode == kModeAllReduce && p.world == 1;
        // tokens this CTA finishes: bit (t >> 2) & 1 set (of a pair, each CTA every other group of four)
        const uint32_t groups = p.csize == 2 ? 1u << crank : 3u;
        const size_t astride = (size_t)p.lay.max_m * p.lay.max_n;
        float *cv_s = reinterpret_cast<float *>(smem + S.cand);        // [EW warps][MP]; a warp fills its own columns
        uint32_t *ci_s = reinterpret_cast<uint32_t *>(smem + S.cand) + EW * MP;
        if (p.mode == kModeLmHead)
            for (int i = lane; i < MP; i += 32) { cv_s[ew * MP + i] = -INFINITY; ci_s[ew * MP + i] = 0xFFFFFFFFu; }

        // A finished tile: its rows go to the output or to the peers; of an lm_head tile the candidates are
        // kept and, when the caller wants them, the logits stored.
        auto finalize = [&](const float (&v)[CP], int tile, const int m, const uint32_t groups) {  // v[i]: token col0 + i
            // columns of the even and of the odd groups that this CTA finishes: one comparison each.  (A predicate for the
            // parity beside the one for m: eight ranks in one launch, three rows 29.2 us a step, 27.1 now, eight 40.4,
            // 38.6; UE8M0 5120 x 2304, 33 to 64 rows, whose sums it spilled, 10.9, 10.5)
            const int even = (groups & 1u) ? m - col0 : 0, odd = (groups & 2u) ? m - col0 : 0;
            auto done = [&](int i) { return i < ((i & 4) ? odd : even); };  // (col0 is a multiple of 16)
            const int row = tile * TR + rc;
            const bool mine = rc < TR && row < p.n;
            // element (token, row) of a float matrix with `ld` floats per token
            // (its stride is hidden from the optimiser, which would keep every column's offset in registers through
            // the main loop: 60 more of them, and spills in the other roles' loops)
            auto store = [&](float *base, int64_t ld) {
                asm volatile("" : "+l"(ld));
                float *dst = base + col0 * ld + row;
#pragma unroll
                for (int i = 0; i < CP; ++i) {
                    if (done(i)) *dst = v[i];
                    dst += ld;
                }
            };
            if (mine) {
                if (solo) {
                    store(A.out, p.n);
                } else if (p.mode == kModeAllReduce) {
                    // every rank gets the partial sums, or (many rows, many ranks) only the tile's owner
                    const int pr0 = p.owner_reduce ? tile % p.world : 0, pr1 = p.owner_reduce ? pr0 + 1 : p.world;
                    for (int pr = pr0; pr < pr1; ++pr) {
                        int64_t ld = p.n;
                        asm volatile("" : "+l"(ld));
                        uint64_t *dst = reinterpret_cast<uint64_t *>(X.sym[pr] + p.lay.slota_off) + ((size_t)bank * p.world + X.rank) * astride + col0 * ld + row;
#pragma unroll
                        for (int i = 0; i < CP; ++i) {
                            if (done(i)) st_word_sys(dst, seq, v[i]);
                            dst += ld;
                        }
                    }
                } else if (p.gather_logits && p.world == 1) {  // a lone rank's logits are final where they are
                    store(A.logits + A.vocab_row0, p.vocab);
                } else if (p.gather_logits) {
                    for (int pr = 0; pr < p.world; ++pr)
                        store(reinterpret_cast<float *>(X.sym[pr] + p.lay.gather_off) + (size_t)bank * p.lay.max_m * (size_t)p.lay.max_vocab +
                                  A.vocab_row0, p.lay.max_vocab);
                }
            }
            if (p.mode == kModeLmHead) {
                // Best (value, lowest index) of this warp's 32 rows per token: the largest key by one redux, the lowest
                // lane that holds it by one ballot, column i's handed to lane i mod 32, so that the columns' chains
                // overlap; each lane then merges its columns into the warp's running best.  (Merged column by column,
                // each a shared-memory round trip behind the last, the accumulators were held up at a tile's end and
                // HBM idled: 64 rows of 62944 x 4352 with logits 94.8 us a step, 82.0 with this, ~65 with the exchange
                // in a function of its own; 32 rows 67.2, 64.2; one row 51.5, 50.9)
                const uint32_t idx0 = (uint32_t)(A.vocab_row0 + tile * TR + quad * 32);
                constexpr int H = (CP + 31) / 32;
                uint32_t best[H], who[H];
#pragma unroll
                for (int h = 0; h < H; ++h) best[h] = who[h] = 0u;
#pragma unroll
                for (int g = 0; g < CP; g += 8) {
                    if (col0 + g >= m) break;  // warp-uniform
#pragma unroll
                    for (int i = g; i < g + 8; ++i) {
                        const uint32_t key = mine ? order_key(v[i]) : 0u;
                        const uint32_t top = __reduce_max_sync(0xffffffffu, key);
                        const uint32_t first = (uint32_t)__ffs(__ballot_sync(0xffffffffu, key == top)) - 1u;
                        if (lane == (i & 31)) { best[i / 32] = top; who[i / 32] = first; }
                    }
                }
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const int c = h * 32 + lane, t = col0 + c;
                    if (c >= CP || !done(c) || best[h] == 0u) continue;
                    const float top = order_value(best[h]);
                    if (cand_better(top, idx0 + who[h], cv_s[ew * MP + t], ci_s[ew * MP + t])) {
                        cv_s[ew * MP + t] = top;
                        ci_s[ew * MP + t] = idx0 + who[h];
                    }
                }
                __syncwarp();
            }
        };

        bool ok = true;
        int ntile_done = 0;
        float acc[CP];
        // positions in the stage and accumulator rings, advanced incrementally
        uint32_t done = done0, ph = 0, accempty = accempty0, t_col = tlane + (uint32_t)col0;
        const uint32_t done_end = done0 + NS * 8, acc_end = accempty0 + NB * 8;
        const int kcta = k_hi - k_lo;
        for (int tile = t_lo; tile <= t_hi && kcta > 0; ++tile) {
#pragma unroll
            for (int i = 0; i < CP; ++i) acc[i] = 0.0f;
            const int row = min(tile * TR + min(rc, TR - 1), p.n - 1);
            const float *swrow = WUE ? nullptr : sw_s + (int)(((A.row0 + row) >> p.bn_shift) - srow_lo) * p.skb;
            int kk = kofs + k_lo * 128;  // K offset of the stage's first slab inside the scale matrix
            for (int left = kcta; left > 0; left -= SL) {
                const int na = (min(left, SL) + CH - 1) / CH;
                if (ok && !mbar_wait(done, ph, X.status)) ok = false;
                ok = __all_sync(0xffffffffu, ok);  // the tensor-memory loads below need the whole warp
                tc_fence_after();
                if (ok) {
                    // as many accumulators per round trip to tensor memory as the registers hold (a last round may
                    // read accumulators of other stages, inside the allocation, and leaves them unused)
                    constexpr int B = bs_read_batch(MP, WUE), C = WUE && CP > 32 ? 32 : CP;  // columns of each
#pragma unroll 1
                    for (int j0 = 0; j0 < na; j0 += B) {
#pragma unroll
                        for (int c = 0; c < CP; c += C) {
                            uint32_t r[B * C];
                            tmem_ld_batch<C, B>(t_col + (uint32_t)(j0 * MP + c), (uint32_t)MP, r);
#pragma unroll
                            for (int j = 0; j < B; ++j)
                                if (j == 0 || j0 + j < na) {
                                    const float sw = WUE ? 1.0f : swrow[(kk + (j0 + j) * 128) >> p.bk_shift];
#pragma unroll
                                    for (int i = 0; i < C; ++i) {
                                        const float v = __uint_as_float(r[j * C + i]);
                                        acc[c + i] = WUE ? acc[c + i] + v : fmaf(v, sw, acc[c + i]);
                                    }
                                }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(accempty);
                kk += SL * 128;
                done += 8;
                if (done == done_end) { done = done0; ph ^= 1u; }
                accempty += 8; t_col += (uint32_t)(AS * MP);
                if (accempty == acc_end) { accempty = accempty0; t_col = tlane + (uint32_t)col0; }
            }
            // what depends on the tile's end only is not worth registers in the main loop: hidden from the optimiser
            int m = p.m, at = col0 / 8 * kBsMmaRows + rc;
            uint32_t gr = groups;
            asm volatile("" : "+r"(gr), "+r"(m), "+r"(at));
            if (p.csize == 2) {
                // a pair swaps its sums: each CTA gets the partner's for the tokens it finishes, in its shared memory
                if (ntile_done > 0) mbar_wait_cluster(rxempty, (uint32_t)(ntile_done - 1) & 1u, X.status);  // the partner has read the previous tile's
                const uint32_t rx = smem_u32(smem + S.rx) + (uint32_t)at * 16u, dst = mapa_u32(rx, crank ^ 1u);
                auto swap = [&](auto mine) {  // K half 0 + K half 1, in that order (the sum of two does not depend on it)
                    constexpr int R = decltype(mine)::value;
#pragma unroll
                    for (int i = 4 * (R ^ 1); i < CP; i += 8)
                        if (col0 + i < m) st_cluster_f32x4(dst + (uint32_t)(i / 8 * kBsMmaRows) * 16u, acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(mapa_u32(rxfull, crank ^ 1u));
                    mbar_wait_cluster(rxfull, (uint32_t)ntile_done & 1u, X.status);
#pragma unroll
                    for (int i = 4 * R; i < CP; i += 8)
                        if (col0 + i < m) {
                            const uint4 v = lds_u128(rx + (uint32_t)(i / 8 * kBsMmaRows) * 16u);
                            acc[i] += __uint_as_float(v.x);
                            acc[i + 1] += __uint_as_float(v.y);
                            acc[i + 2] += __uint_as_float(v.z);
                            acc[i + 3] += __uint_as_float(v.w);
                        }
                };
                if (gr == 1u) swap(std::integral_constant<int, 0>{});
                else swap(std::integral_constant<int, 1>{});
                __syncwarp();
                if (lane == 0 && tile < t_hi) mbar_arrive_cluster(mapa_u32(rxempty, crank ^ 1u));  // nobody waits for the last one
            }
            finalize(acc, tile, m, gr);
            ++ntile_done;
        }
    }

    // ---- teardown: every TMEM read and MMA has completed once all threads are here
    tc_fence_before();
    __syncthreads();
    if (p.csize == 2) {  // neither CTA of a pair leaves while the other may still write to or signal it
        // What each sent was waited for by the other, so neither need wait for its own output stores to reach
        // memory (a release would: ~1 us).
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
    if (p.world > 1 && p.mode == kModeAllReduce) bs_fold(p, EW, CP);
    if (p.mode == kModeLmHead) bs_lm_head<MP, WUE, INL>(p);
    if (p.world > 1 || p.mode == kModeLmHead) step_end(X, step_begin(X), gridDim.x);
    host_done_signal(X, gridDim.x);
}

}  // namespace ws

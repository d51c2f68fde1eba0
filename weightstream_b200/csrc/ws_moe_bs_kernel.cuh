// MXFP4 routed-expert down projection + top-k combine fused with its exchange on the 5th-generation
// tensor cores (sm_100a): tcgen05.mma.kind::mxf8f6f4.block_scale computes exactly this step's product,
// E2M1 weights x E4M3 activations with a UE8M0 scale per 32 values on BOTH operands, so a pass
// accumulates over all of K in tensor memory and the SMs only move bytes.
//
// Two kernels per step:
//
//   moe_bs_prep_kernel  one block per route: its position among the rank's routes sorted by expert
//                       (a pass = one local expert with up to 16 of its routes as MMA columns, experts
//                       in ascending id as crates/weightstream-ref/src/moe.rs:75-84 adds them),
//                       hidden x routing-weight quantised as the reference does (moe.rs:150, then
//                       actquant.rs:21-57) into the form the MMA reads: per pass 16-byte chunks of K,
//                       chunk-major ([chunk][route of the pass][16 bytes]), and the per-32 exponents as the
//                       pass's scale atoms (one per 128-wide K slab, a row of 16 bytes per route: byte j =
//                       exponent of K block j).
//   moe_bs_kernel       persistent CTA pairs (clusters of 2), one pair per tile of ~97 output rows,
//                       each CTA of a pair streams half of K of every pass: with a lone CTA's ~48
//                       rows under half of the MMA's 128 rows would be real, and the tensor pipe
//                       needs the same ~35 ns per K=32 MMA however few are.  Warp 0 lane 0 streams,
//                       per stage of several 128-wide K slabs, the expert's rows (TMA, 4-bit codes
//                       unpacked by the copy into the 16-bytes-per-16-codes form the MMA reads) and the
//                       pass's activations and scale atoms (one bulk copy each, only of the routes there
//                       are: padded to the MMA's 16 columns they were 40 % of the weights' bytes, and what
//                       L2 can hand the SMs bound the step).  Four warps turn the
//                       weights' UE8M0 bytes (4 consecutive bytes per row and slab in the reference's
//                       [expert][row][k/32] layout) into scale atoms in shared memory, one pass ahead.
//                       Warp 1 lane 0 copies both atoms of a slab into tensor memory and issues its
//                       four MMAs; one commit per stage frees it, one per pass hands the accumulator
//                       (16 columns, double-buffered) to the four epilogue warps, which add column t
//                       to the tensor-memory sums of the token that route belongs to.  After the last
//                       pass the CTAs of a pair swap their sums through distributed shared memory, each
//                       adds the halves of K for half of the tokens and stores or exchanges those rows.
//
// A step of up to kMoeBsInlineRoutes routes has no prep kernel: every CTA reads the route ids, makes the pass
// table and quantises its K half of the routes' hidden into shared memory while the weights stream (the prep
// kernel's launch, run and completion stood in front of the first weight byte: ~3 us of a one-token step).
//
// Exchange: as in the FP8 kernels (partials stored to every peer as tagged words, folded in rank order).
#pragma once

#include <math.h>

#include "ws_device.cuh"
#include "ws_fp8_bs_kernel.cuh"      // tcgen05 / cluster wrappers, kBsAtomBytes, kBsMmaRows
#include "ws_moe_gemv_kernel.cuh"    // MoePass, kMoeMaxRoutes, kMoeMaxExperts

namespace ws {

constexpr int kMoeBsCols = 16;        // routes of one expert per pass = N of the MMA
constexpr int kMoeBsThreads = 320;    // warp 0 producer, 1 MMA issue, 2-5 epilogue, 6-9 weight-scale atoms
constexpr int kMoeBsInlineRoutes = 16;  // up to so many routes the main kernel sorts and quantises itself (no prep launch)
constexpr int kMoeBsMaxSlabs = 16;    // K slabs one CTA walks per pass (k <= 4096 with pairs)

// Per-endpoint scratch written by moe_bs_prep_kernel and read by moe_bs_kernel.
struct MoeBsWork {
    int64_t hdr, pass, stok, xq, total;  // byte offsets
};
__host__ __device__ inline MoeBsWork moe_bs_work_layout(int k) {
    MoeBsWork w{};
    int64_t o = 0;
    w.hdr = o;  o += 64;
    w.pass = o; o += (int64_t)kMoeMaxRoutes * sizeof(MoePass);
    w.stok = o; o += align_up((int64_t)(kMoeMaxRoutes + kMoeBsCols) * 2, 256);
    // a pass starts at its first route's share; per K half and group of up to SL slabs: [8 * slabs chunks][nr][16],
    // then the group's atoms [slabs][nr][16]
    w.xq = o;   o += (int64_t)kMoeMaxRoutes * (k / 128) * 144;
    w.total = o;
    return w;
}

struct MoeBsPrepParams {
    int32_t m, k, top_k, h_dtype, sl, pad0;
    MoePrepRank r[WS_MAX_WORLD];
};

__device__ __forceinline__ int block_sum_256(int v, int *red_s) {  // all 256 threads get the sum
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red_s[warp] = v;
    __syncthreads();
    int s = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red_s[w];
    return s;
}

__global__ void __launch_bounds__(256) moe_bs_prep_kernel(const __grid_constant__ MoeBsPrepParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const MoePrepRank &A = p.r[blockIdx.y];
    const int NR = p.m * p.top_k, tid = threadIdx.x;
    // The route's hidden row, asked for before it is known to be this rank's.  (Without and with, 48 of 384 experts on this
    // rank: 8 tokens of 5120 x 2304 16.65 us a step, 16.3; 21 of 7168 x 2048 30.6, 30.3; 64 54.6, 54.2; all experts, no
    // difference.)
    if ((int)blockIdx.x < NR)
        for (int c = tid; c < (p.k >> 4); c += blockDim.x) prefetch_act(A.h, p.h_dtype, (int64_t)blockIdx.x * A.ldh + c * 16);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const MoeBsWork W = moe_bs_work_layout(p.k);
    __shared__ int32_t cnt_s[kMoeMaxExperts];
    __shared__ int red_s[8];
    for (int i = tid; i < A.e_len; i += blockDim.x) cnt_s[i] = 0;
    __syncthreads();
    for (int i = tid; i < NR; i += blockDim.x) {
        const int e = A.route_ids[i] - A.e_start;
        if (e >= 0 && e < A.e_len) atomicAdd(&cnt_s[e], 1);
    }
    __syncthreads();
    if ((int)blockIdx.x == NR) {  // the extra block: how many passes the step has
        int np = 0;
        for (int e = tid; e < A.e_len; e += blockDim.x) np += (cnt_s[e] + kMoeBsCols - 1) / kMoeBsCols;
        np = block_sum_256(np, red_s);
        if (tid == 0) *reinterpret_cast<int32_t *>(A.work + W.hdr) = np;
        return;
    }
    const int route = blockIdx.x;
    const int e = A.route_ids[route] - A.e_start;
    if (e < 0 || e >= A.e_len) return;  // another rank's expert (or none)
    // position among the rank's routes sorted by (expert, route), rank among the expert's routes,
    // and the passes of the experts before this one
    int pos = 0, rnk = 0, pb = 0;
    for (int i = tid; i < NR; i += blockDim.x) {
        const int ei = A.route_ids[i] - A.e_start;
        if (ei < 0 || ei >= A.e_len) continue;
        if (ei < e || (ei == e && i < route)) ++pos;
        if (ei == e && i < route) ++rnk;
    }
    for (int i = tid; i < e; i += blockDim.x) pb += (cnt_s[i] + kMoeBsCols - 1) / kMoeBsCols;
    pos = block_sum_256(pos, red_s);
    rnk = block_sum_256(rnk, red_s);
    pb = block_sum_256(pb, red_s);
    const int pass = pb + rnk / kMoeBsCols, t = rnk % kMoeBsCols;
    if (tid == 0) {
        if (t == 0) {
            MoePass ps;
            ps.expert = (uint16_t)e;
            ps.first = (uint16_t)pos;
            ps.nr = (uint16_t)min(kMoeBsCols, cnt_s[e] - rnk);
            ps.pad = 0;
            reinterpret_cast<MoePass *>(A.work + W.pass)[pass] = ps;
        }
        reinterpret_cast<uint16_t *>(A.work + W.stok)[pos] = (uint16_t)(route / p.top_k);
    }
    const float w = A.route_w[route];
    const int first = pos - t, nr = min(kMoeBsCols, cnt_s[e] - (rnk - t));  // the pass's first route and route count
    uint8_t *xq = A.work + W.xq + (size_t)first * (p.k >> 7) * 144;
    for (int c = tid; c < (p.k >> 4); c += blockDim.x) {  // the two chunks of a 32-block are adjacent lanes
        float v[16];
        load_act8(A.h, p.h_dtype, (int64_t)route * A.ldh + c * 16, true, *reinterpret_cast<float(*)[8]>(v));
        load_act8(A.h, p.h_dtype, (int64_t)route * A.ldh + c * 16 + 8, true, *reinterpret_cast<float(*)[8]>(v + 8));
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] *= w;
        int ex;
        const uint4 q = act_quant16(v, ex);
        int count;
        const int slab = c >> 3, g0 = bs_group(slab, p.k >> 7, 2, p.sl, count);
        uint8_t *grp = xq + (size_t)g0 * nr * 144;
        *reinterpret_cast<uint4 *>(grp + ((size_t)(c - g0 * 8) * nr + t) * 16) = q;
        if ((c & 1) == 0) grp[(size_t)count * nr * 128 + ((size_t)(slab - g0) * nr + t) * 16 + ((c >> 1) & 3)] = (uint8_t)min(max(ex + 127, 0), 255);
    }
}

// ------------------------------------------------------------------------------------------
struct MoeBsRank {
    const uint8_t *s2;    // [e_len][n][k/32] UE8M0
    const uint8_t *work;  // MoeBsWork
    float *out;           // [m][n]
    const void *h;        // inline form only: hidden, route ids and weights as the prep kernel takes them
    const int32_t *route_ids;
    const float *route_w;
    int64_t ldh;
    int32_t e_start, e_len;
    RankCtx ctx;
};

struct alignas(64) MoeBsParams {
    // expert slab as [e_len][k / 128][n][128] 4-bit codes; boxes of 128 codes x tile_rows x SL slabs ([0]) or one
    // slab ([t]: those of a group that is not whole), unpacked, 128B swizzle
    CUtensorMap tmap_w[WS_MAX_WORLD], tmap_t[WS_MAX_WORLD];
    int32_t m, n, k, world;
    int32_t tile_rows, a_pitch, slabs_per_stage, nstages;
    int32_t tmem_cols, x_pitch, alias, nroutes;  // alias: the partner's sums land in the ring; nroutes = m * top_k
    int32_t inline_x, top_k, h_dtype, pad0;
    uint64_t timeout_ns;
    SymLayout lay;
    MoeBsRank r[WS_MAX_WORLD];
};

struct MoeBsSmem {
    int32_t a, b, sfa, rx, pass, tok, bars, misc, total;
};
__host__ __device__ inline MoeBsSmem moe_bs_smem_layout(int nstages, int slabs_per_stage, int a_pitch, int x_pitch, int m, int nslab_cta,
                                                        int alias, int nroutes, int inline_x) {
    MoeBsSmem s{};
    int o = 0;
    s.a = o;    o += nstages * slabs_per_stage * a_pitch;
    // per stage: its slabs' activations, then their scale atoms; inline: those of all routes, this K half
    const int b_bytes = inline_x ? nroutes * nslab_cta * 144 : nstages * x_pitch;
    s.b = o;    o += (b_bytes + 127) / 128 * 128;
    // an MMA reads 128 rows behind the last weight slab, 16 routes and 32 atom rows whatever the pass has
    o += b_bytes + 2048 < kBsMmaRows * 128 ? kBsMmaRows * 128 - b_bytes / 128 * 128 : 2048;
    s.sfa = o;  o += 2 * nslab_cta * kBsAtomBytes;                      // weight-scale atoms of two passes
    s.rx = alias ? 0 : o;                                               // the partner's, at the end
    o += alias ? 0 : (m + 1) / 2 * kBsMmaRows * 4;
    s.pass = o; o += (nroutes * (int)sizeof(MoePass) + 15) / 16 * 16;
    s.tok = o;  o += ((nroutes > kMoeBsInlineRoutes ? nroutes : 2 * kMoeBsInlineRoutes) * 2 + 15) / 16 * 16;
    s.bars = o; o += (2 * kMaxStages + 12) * 8;
    s.misc = o; o += 128;
    s.total = o;
    return s;
}

// Instruction descriptor: E2M1 weights (format code 5) x E4M3 activations, UE8M0 scales, M = 128, N = 16.
__device__ __forceinline__ uint32_t moe_bs_idesc(int sf_id) {
    return ((uint32_t)sf_id << 4) | (5u << 7) | (0u << 10) | ((uint32_t)(kMoeBsCols >> 3) << 17) | (1u << 23) | (8u << 24) |
           ((uint32_t)sf_id << 29);
}

// Inline form: the 256 threads of warps 2-9 quantise hidden x routing-weight of this CTA's K half into the
// resident activation area: per pass [chunk][nr][16 bytes], then, after those of all routes, the scale atoms.
// The first two rounds' values (all there are in a one-token step) are loaded before the table is there.
__device__ __forceinline__ void moe_bs_quantise(const MoeBsParams &p, const MoeBsRank &A, uint8_t *xres, const uint16_t *place,
                                                int nslab, int k_lo, int t256) {
    const int chunks = nslab * 8, total = p.nroutes * chunks;  // two adjacent lanes share a 32-block
    uint8_t *atoms = xres + (size_t)p.nroutes * chunks * 16;
    for (int c0 = t256; c0 - (t256 & 31) < total; c0 += 512) {  // whole warps
        float v[2][16], w[2];
        int rt[2], ch[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = c0 + u * 256;
            const bool in = c < total;
            rt[u] = in ? c / chunks : 0;
            ch[u] = in ? c - rt[u] * chunks : 0;
            const int64_t at = (int64_t)rt[u] * A.ldh + (int64_t)k_lo * 128 + ch[u] * 16;
            load_act8(A.h, p.h_dtype, at, in, *reinterpret_cast<float(*)[8]>(v[u]));
            load_act8(A.h, p.h_dtype, at + 8, in, *reinterpret_cast<float(*)[8]>(v[u] + 8));
            w[u] = in ? A.route_w[rt[u]] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[u][i] *= w[u];
            int ex;
            const uint4 q = act_quant16(v[u], ex);
            const int pl = place[rt[u]], first = pl & 31, t = pl >> 5 & 31, nr = pl >> 10;
            if (c0 + u * 256 < total && nr > 0) {
                *reinterpret_cast<uint4 *>(xres + ((size_t)first * chunks + (size_t)ch[u] * nr + t) * 16) = q;
                if ((ch[u] & 1) == 0)
                    atoms[((size_t)first * nslab + (size_t)(ch[u] >> 3) * nr + t) * 16 + ((ch[u] >> 1) & 3)] = (uint8_t)min(max(ex + 127, 0), 255);
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// One tensor-memory column of this warp's lanes.
__device__ __forceinline__ float tmem_ld_one(uint32_t taddr) {
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\ttcgen05.wait::ld.sync.aligned;" : "=r"(r) : "r"(taddr) : "memory");
    return __uint_as_float(r);
}
__device__ __forceinline__ void tmem_st_one(uint32_t taddr, float v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(__float_as_uint(v)) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 4-D TMA tile load (codes, rows, slab, expert), completion on an mbarrier.
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, int w, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}

__global__ void __launch_bounds__(kMoeBsThreads, 1) moe_bs_kernel(const __grid_constant__ MoeBsParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);

    const int vr = blockIdx.y, cta = blockIdx.x, ncta = gridDim.x;
    const MoeBsRank &A = p.r[vr];
    const RankCtx &X = A.ctx;
    const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
    uint32_t crank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    const int part = cta >> 1, TR = p.tile_rows;
    const int row0 = part * TR;                                     // this pair's rows [row0, row0 + TR)
    const int KS = p.k >> 7;
    const int k_lo = (int)crank * KS / 2, k_hi = ((int)crank + 1) * KS / 2;
    const int NSLAB = k_hi - k_lo;                                  // slabs this CTA walks per pass
    const int SL = p.slabs_per_stage, NS = p.nstages;
    const int IP = (NSLAB + SL - 1) / SL;                           // stage items per pass

    const MoeBsSmem S = moe_bs_smem_layout(NS, SL, p.a_pitch, p.x_pitch, p.m, NSLAB, p.alias, p.nroutes, p.inline_x);
    const MoeBsWork W = moe_bs_work_layout(p.k);
    uint32_t *misc_s = reinterpret_cast<uint32_t *>(smem + S.misc);
    const uint32_t a0 = smem_u32(smem + S.a), b0 = smem_u32(smem + S.b), sfa0 = smem_u32(smem + S.sfa);
    // full[s]: a stage's bytes landed; done[s]: its MMAs have completed (stage free), except for the last stage
    // of a pass, where accfull says so too (a second commit right behind the first waits for the first's MMAs);
    // accfull[pass mod 4] / accempty[g]: a pass's accumulator is complete (and its scale columns free again) /
    // has been read; sfafull[g]: the weight scales of a pass are in tensor memory.
    const uint32_t full0 = smem_u32(smem + S.bars), done0 = full0 + kMaxStages * 8;
    const uint32_t accfull0 = done0 + kMaxStages * 8, accempty0 = accfull0 + 32, sfafull0 = accempty0 + 16;
    const uint32_t xready = sfafull0 + 16;  // inline: the routes' activations are in shared memory

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full0 + s * 8, 1);
            mbar_init(done0 + s * 8, 1);
        }
        for (int b = 0; b < 4; ++b) mbar_init(accfull0 + b * 8, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(accempty0 + b * 8, 4);    // one arrival per epilogue warp
            mbar_init(sfafull0 + b * 8, 1);     // the commit that follows the scale warps' copies
        }
        mbar_init(xready, 256);
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(misc_s), (uint32_t)p.tmem_cols);
        tmem_relinquish();
    }
    if (tid == 0) misc_s[8] = 0u;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(misc_s);
    // tensor-memory columns: two accumulators of 16, per pass buffer and slab 4 activation-scale and 4
    // weight-scale columns, then the sums of every token (lane = row): in shared memory those of 64 tokens took
    // 32 KB from the ring, and the step was bound by the bytes in flight
    const uint32_t t_sc0 = tmem_base + 2u * kMoeBsCols, t_tok0 = t_sc0 + (uint32_t)(2 * NSLAB * 8);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // everything below depends on the routes (or the prep kernel's pass table)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    MoePass *passes = reinterpret_cast<MoePass *>(smem + S.pass);
    uint16_t *stok = reinterpret_cast<uint16_t *>(smem + S.tok);  // token of every route, sorted by (expert, route)
    int npass;
    if (p.inline_x) {
        // One pass per expert (at most 16 routes).  Lane = route, every warp for itself: the lanes of the same
        // expert by one match, a route's place by counting the routes before it in (expert, route) order.
        const int e = lane < p.nroutes ? A.route_ids[lane] - A.e_start : -1;
        const bool local = e >= 0 && e < A.e_len;
        const uint32_t valid = __ballot_sync(0xffffffffu, local);
        const uint32_t same = __match_any_sync(0xffffffffu, local ? e : -1 - lane);
        const uint32_t leaders = __ballot_sync(0xffffffffu, local && (same & ((1u << lane) - 1u)) == 0u);
        npass = __popc(leaders);
        if (warp == 0) {
            int below = 0, before = 0;  // routes and passes of smaller experts
#pragma unroll
            for (int i = 0; i < kMoeBsInlineRoutes; ++i) {
                const int ei = __shfl_sync(0xffffffffu, e, i);
                const bool less = (valid >> i & 1u) && ei < e;
                below += less ? 1 : 0;
                before += less && (leaders >> i & 1u) ? 1 : 0;
            }
            if (local) {
                const int t = __popc(same & ((1u << lane) - 1u)), pos = below + t;
                if (t == 0) passes[before] = MoePass{(uint16_t)e, (uint16_t)below, (uint16_t)__popc(same), (uint16_t)0};
                stok[pos] = (uint16_t)(lane / p.top_k);
                // for the quantiser, by route: its pass's first place and count, its own place in the pass (the
                // token table has room for 16 more entries)
                stok[kMoeBsInlineRoutes + lane] = (uint16_t)(below | t << 5 | __popc(same) << 10);
            } else if (lane < p.nroutes) {
                stok[kMoeBsInlineRoutes + lane] = 0;  // another rank's
            }
        }
    } else {
        npass = *reinterpret_cast<const volatile int32_t *>(A.work + W.hdr);
        const MoePass *src = reinterpret_cast<const MoePass *>(A.work + W.pass);
        for (int i = tid; i < npass; i += kMoeBsThreads) passes[i] = src[i];
        const uint16_t *st = reinterpret_cast<const uint16_t *>(A.work + W.stok);
        for (int i = tid; i < p.nroutes; i += kMoeBsThreads) stok[i] = st[i];
    }
    __syncthreads();

    if (warp == 0) {
        // ------------------------------------------------------------ producer (one thread)
        if (elect_one()) {
            RingPos st;
            int item = 0, pp = 0, pi = 0;
            uint32_t done_ph = 0;  // per stage: parity of the next completion of done[s]
            for (int ps = 0; ps < npass; ++ps) {
                const MoePass P = passes[ps];
                const uint32_t x_slab = (uint32_t)P.nr * 144u;
                const uint8_t *xq = A.work + W.xq + (size_t)P.first * KS * 144 + (size_t)k_lo * x_slab;
                for (int i = 0; i < IP; ++i, ++item, st.next(NS)) {
                    const int s = st.s, j0 = i * SL, nsl = min(SL, NSLAB - j0);
                    if (item >= NS) {  // the stage's previous item, number pi of pass pp, has been read
                        const bool freed = pi == IP - 1 ? mbar_wait(accfull0 + (pp & 3) * 8, (uint32_t)(pp >> 2) & 1u, X.status)
                                                        : mbar_wait(done0 + s * 8, done_ph >> s & 1u, X.status);
                        if (!freed) { ps = npass; break; }
                        if (pi == IP - 1) { pi = 0; ++pp; }
                        else { ++pi; done_ph ^= 1u << s; }
                    }
                    // the unpacking copy counts the packed bytes it read (64 per row), not the 128 it wrote
                    mbar_arrive_expect_tx(full0 + s * 8, (uint32_t)nsl * ((uint32_t)TR * 64u + (p.inline_x ? 0u : x_slab)));
                    const uint32_t dst = a0 + s * SL * p.a_pitch;
                    if (nsl == SL) {
                        tma_load_4d(dst, &p.tmap_w[vr], 0, row0, k_lo + j0, (int)P.expert, full0 + s * 8);
                    } else {
                        for (int j = 0; j < nsl; ++j) tma_load_4d(dst + j * p.a_pitch, &p.tmap_t[vr], 0, row0, k_lo + j0 + j, (int)P.expert, full0 + s * 8);
                    }
                    if (!p.inline_x) bulk_load(b0 + s * p.x_pitch, xq + (size_t)j0 * x_slab, (uint32_t)nsl * x_slab, full0 + s * 8);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issue (one thread)
        if (elect_one()) {
            // As in the FP8 kernel, what stands between two stages' MMAs has to stay short.
            const uint32_t id0 = moe_bs_idesc(0), id1 = moe_bs_idesc(1), id2 = moe_bs_idesc(2), id3 = moe_bs_idesc(3);
            uint32_t *const status = X.status;
            const bool inl = p.inline_x != 0;
            const uint32_t a_lo0 = umma_desc_lo(a0), b_lo0 = (b0 & 0x3FFFFu) >> 4;
            const uint32_t a_stage = (uint32_t)(SL * p.a_pitch) >> 4, x_stage = (uint32_t)p.x_pitch >> 4;
            const uint32_t whole_step = (uint32_t)TR * 8u, part_step = (uint32_t)p.a_pitch >> 4;  // slabs of one box follow row by row
            const uint64_t sf_desc0 = umma_desc(b0, 128, false);
            const uint32_t sf_inl = (uint32_t)(p.nroutes * NSLAB) * 8u;
            uint32_t full = full0, done = done0, a_lo = a_lo0, x_off = 0, ph = 0;
            const uint32_t full_end = full0 + NS * 8;
            bool ok = !inl || mbar_wait(xready, 0, status);
            MoePass P = npass > 0 ? passes[0] : MoePass{};
            for (int ps = 0; ps < npass && ok; ++ps) {
                const uint32_t g = (uint32_t)ps & 1u, lap = (uint32_t)(ps >> 1) & 1u;
                const uint32_t t_acc = tmem_base + g * kMoeBsCols;
                uint32_t t_sc = t_sc0 + g * (uint32_t)(NSLAB * 8);
                const uint32_t nr = P.nr, b_step = 8u * nr, x_kb = 2u * nr;  // 16-byte units
                // inline: the pass's activations and atoms in the resident area, else a stage's, atoms after activations
                uint32_t x_in = (uint32_t)P.first * (uint32_t)NSLAB * 8u, sf_in = sf_inl + (uint32_t)P.first * (uint32_t)NSLAB;
                uint32_t acc = 0;
                if (!mbar_wait(accempty0 + g * 8, lap ^ 1u, status) || !mbar_wait(sfafull0 + g * 8, lap, status)) break;
                for (int left = NSLAB; left > 0; left -= SL) {
                    if (!mbar_wait(full, ph, status)) { ok = false; break; }
                    tc_fence_after();
                    const int nsl = min(left, SL);
                    const uint32_t a_step = nsl == SL ? whole_step : part_step;
                    uint32_t a = a_lo, b = (b_lo0 + (inl ? x_in : x_off)) | (nr << 16);
                    uint64_t sf = sf_desc0 + (uint64_t)(inl ? sf_in : x_off + (uint32_t)nsl * b_step);
                    // straight-line code, four slabs at a time
                    auto issue = [&](auto count) {
                        constexpr int C = decltype(count)::value;
#pragma unroll
                        for (int j = 0; j < C; ++j) {
                            const uint32_t aj = a + (uint32_t)j * a_step, bj = b + (uint32_t)j * b_step, sx = t_sc + (uint32_t)(j * 8);
                            tmem_cp_atom(sx, sf + (uint64_t)((uint32_t)j * nr));  // the activations' scales of this slab (the weights' are there already)
                            umma_bs_ss(t_acc, aj, bj, kUmmaDescHiSw128, kUmmaDescHiX, id0, sx + 4, sx, j > 0 ? 1u : acc);
                            umma_bs_ss(t_acc, aj + 2, bj + x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id1, sx + 4, sx, 1u);
                            umma_bs_ss(t_acc, aj + 4, bj + 2 * x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id2, sx + 4, sx, 1u);
                            umma_bs_ss(t_acc, aj + 6, bj + 3 * x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id3, sx + 4, sx, 1u);
                        }
                        acc = 1;
                        a += (uint32_t)C * a_step; b += (uint32_t)C * b_step; sf += (uint64_t)((uint32_t)C * nr); t_sc += C * 8;
                    };
                    int n4 = nsl;
                    for (; n4 >= 4; n4 -= 4) issue(std::integral_constant<int, 4>{});
                    if (n4 == 3) issue(std::integral_constant<int, 3>{});
                    else if (n4 == 2) issue(std::integral_constant<int, 2>{});
                    else if (n4 == 1) issue(std::integral_constant<int, 1>{});
                    // the stage may be refilled (and, at the end of the pass, its sums are complete and its scale columns free)
                    umma_commit(left <= SL ? accfull0 + ((uint32_t)ps & 3u) * 8u : done);
                    x_in += (uint32_t)SL * b_step; sf_in += (uint32_t)SL * nr;
                    full += 8; done += 8; a_lo += a_stage; x_off += x_stage;
                    if (full == full_end) {
                        full = full0; done = done0; a_lo = a_lo0; x_off = 0;
                        ph ^= 1u;
                    }
                }
                if (ps + 1 < npass) P = passes[ps + 1];
            }
        }
        __syncwarp();
    } else if (warp >= 6) {
        // ------------------------------------------------------------ weight scales, one pass ahead
        // The expert's UE8M0 bytes of this CTA's rows and K half become scale atoms in shared memory
        // (thread = row), and one thread copies them into the pass's tensor-memory columns: the
        // MMA-issuing thread only waits for that commit.
        const int r = tid - 192;  // 0..127: row of the tile = lane of the atom
        const int row = row0 + r;
        const bool real = r < TR && row < p.n;
        const int kb32 = p.k >> 5;
        const uint64_t sfa_desc0 = umma_desc(sfa0, 128, false);
        uint32_t sc[kMoeBsMaxSlabs];  // the next pass's bytes, on their way while this one is written
        auto fetch = [&](int ps) {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(A.s2 + ((size_t)passes[ps].expert * p.n + (real ? row : 0)) * kb32) + k_lo;
#pragma unroll
            for (int j = 0; j < kMoeBsMaxSlabs; ++j)
                if (j < NSLAB) sc[j] = real ? __ldg(src + j) : 0x7F7F7F7Fu;
        };
        if (npass > 0) fetch(0);
        if (p.inline_x) {
            moe_bs_quantise(p, A, smem + S.b, stok + kMoeBsInlineRoutes, NSLAB, k_lo, tid - 64);
            mbar_arrive(xready);
        }
        for (int ps = 0; ps < npass; ++ps) {
            const int g = ps & 1;
            const uint32_t lap = (uint32_t)(ps >> 1) & 1u;
            // the pass that used these columns and this buffer last (ps - 2) has completed; a wait that
            // gave up is told to all four warps at the barrier below, so that they leave the loop together
            if (ps >= 2 && !mbar_wait(accfull0 + ((ps - 2) & 3) * 8, (uint32_t)((ps - 2) >> 2) & 1u, X.status)) misc_s[8] = 1u;
            uint8_t *dst = smem + S.sfa + (size_t)(g * NSLAB) * kBsAtomBytes + (r & 31) * 16 + (r >> 5) * 4;
#pragma unroll
            for (int j = 0; j < kMoeBsMaxSlabs; ++j)
                if (j < NSLAB) *reinterpret_cast<uint32_t *>(dst + (size_t)j * kBsAtomBytes) = sc[j];
            if (ps + 1 < npass) fetch(ps + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("bar.sync 3, 128;" ::: "memory");
            if (*reinterpret_cast<volatile uint32_t *>(misc_s + 8) != 0u) break;
            if (warp == 6 && elect_one()) {
                tc_fence_after();
                const uint32_t t_sfa = t_sc0 + (uint32_t)(g * NSLAB * 8) + 4u;
                const uint64_t sfa_desc = sfa_desc0 + (uint64_t)((uint32_t)(g * NSLAB) * ((uint32_t)kBsAtomBytes >> 4));
#pragma unroll 4
                for (int j = 0; j < NSLAB; ++j) tmem_cp_atom(t_sfa + (uint32_t)(j * 8), sfa_desc + (uint64_t)((uint32_t)j * ((uint32_t)kBsAtomBytes >> 4)));
                umma_commit(sfafull0 + g * 8);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue warps 2-5
        const int quad = warp & 3;
        const int rc = quad * 32 + lane;  // row inside the tile = TMEM lane
        const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16), t_tok = t_tok0 - tmem_base;
        if (p.inline_x) {
            moe_bs_quantise(p, A, smem + S.b, stok + kMoeBsInlineRoutes, NSLAB, k_lo, tid - 64);
            mbar_arrive(xready);
        }
        for (int t = 0; t < p.m; ++t) tmem_st_one(tlane + t_tok + (uint32_t)t, 0.0f);
        tmem_wait_st();
        bool ok = true;
        for (int ps = 0; ps < npass; ++ps) {
            const int g = ps & 1;
            const uint32_t lap = (uint32_t)(ps >> 1) & 1u;
            const MoePass P = passes[ps];
            if (ok && !mbar_wait(accfull0 + (ps & 3) * 8, (uint32_t)(ps >> 2) & 1u, X.status)) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            uint32_t v[kMoeBsCols];
            tmem_ld_cols<kMoeBsCols>(tlane + (uint32_t)(g * kMoeBsCols), v);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty0 + g * 8);
#pragma unroll
            for (int t = 0; t < kMoeBsCols; ++t)
                if (t < (int)P.nr) {  // in route order: two routes of one pass may belong to one token
                    const uint32_t at = tlane + t_tok + (uint32_t)stok[P.first + t];
                    tmem_st_one(at, tmem_ld_one(at) + __uint_as_float(v[t]));
                    tmem_wait_st();
                }
        }
        tc_fence_before();
    }

    // ---- the pair's halves of K: each CTA sends the other the sums of the tokens that one finishes
    tc_fence_before();
    __syncthreads();
    float *rx_s = reinterpret_cast<float *>(smem + S.rx);
    if (p.alias) {  // the partner's ring is idle: its copies have landed and its MMAs have completed
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    const int split = (p.m + 1) / 2;
    const int tok_lo = crank == 0 ? 0 : split, tok_hi = crank == 0 ? split : p.m;
    const int quad = warp & 3, rc = quad * 32 + lane, row = row0 + rc;  // the epilogue warps: row = TMEM lane
    const uint32_t tlane = t_tok0 + ((uint32_t)(quad * 32) << 16);
    const bool epi = warp >= 2 && warp < 6;
    if (epi) {
        tc_fence_after();
        const int lo = crank == 0 ? split : 0, hi = crank == 0 ? p.m : split;  // the partner's tokens
        const uint32_t dst = mapa_u32(smem_u32(rx_s) + (uint32_t)rc * 4u, crank ^ 1u);
        for (int t = lo; t < hi; ++t) st_cluster_f32(dst + (uint32_t)((t - lo) * kBsMmaRows * 4), tmem_ld_one(tlane + (uint32_t)t));
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // nothing crosses the pair after this

    const bool solo = p.world == 1;
    const bool mine = rc < TR && row < p.n;
    if (epi) {
        const uint32_t seq = step_begin(X);
        const uint32_t bank = seq & 1u;
        const size_t astride = (size_t)p.lay.max_m * p.lay.max_n;
        for (int t = tok_lo; t < tok_hi; ++t) {  // K half 0 + K half 1
            const float v = tmem_ld_one(tlane + (uint32_t)t) + rx_s[(t - tok_lo) * kBsMmaRows + rc];
            if (!mine) continue;
            if (solo) {
                A.out[(size_t)t * p.n + row] = v;
            } else {
                for (int pr = 0; pr < p.world; ++pr) {
                    uint64_t *dstw = reinterpret_cast<uint64_t *>(X.sym[pr] + p.lay.slota_off) + ((size_t)bank * p.world + X.rank) * astride;
                    st_word_sys(dstw + (size_t)t * p.n + row, seq, v);
                }
            }
        }
        if (!solo && mine) {  // fold the same rows in rank order as the ranks' words arrive
            const uint64_t *slots = reinterpret_cast<const uint64_t *>(X.sym[X.rank] + p.lay.slota_off) + (size_t)bank * p.world * astride;
            for (int t = tok_lo; t < tok_hi; ++t) {
                const size_t off = (size_t)t * p.n + row;
                A.out[off] = fold_words(slots, astride, off, p.world, seq, p.timeout_ns, X.status, kStatTimeoutPeerA);
            }
        }
    }

    // ---- teardown
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
    if (p.world > 1) step_end(X, step_begin(X), gridDim.x);
}

}  // namespace ws

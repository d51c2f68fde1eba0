// FP8 E4M3 row-parallel decode GEMM fused with its exchange (sm_100a).
//
// One persistent CTA per SM.  Every output row is a complete dot product inside ONE CTA:
// a CTA owns floor(n/16/ncta) whole 16-row tiles plus a ragged share (at most 16 rows) of the
// rows that are left over, so all SMs stream the same number of bytes and nothing is combined
// across CTAs.  Weight tiles arrive by TMA into a ring of 32 KB stages filled by one producer
// warp: 16-row x 128-byte boxes for whole tiles, 8/4/2/1-row boxes for the ragged rows, all
// 128B-swizzled.  The prologue quantises the activations exactly as the reference does; eight
// consumer warps then multiply the staged rows with them by the FP8 tensor-core MMA m16n8k32, one per
// 32-wide K block, and apply the activation- and weight-block scales in fp32.  Its issue rate caps
// streaming near 70 % of HBM bandwidth: it serves the shapes neither the one- and two-row kernel
// (ws_fp8_gemv_kernel.cuh) nor the tensor-memory kernel (ws_fp8_bs_kernel.cuh) takes.
//
// Exchange (world > 1): a thread stores its rows' fp32 partials into slot [my rank] of every
// peer's exchange memory as 64-bit {step, value} words and then adds the same rows' words of all
// ranks in rank order as they arrive, so all ranks produce identical bits.
//
// lm_head mode: rows are vocabulary entries; instead of a sum every rank's rows are gathered
// (stored into every peer's logits buffer) and each CTA publishes its best (value, lowest
// index) candidate per token; CTA 0 merges them.
#pragma once

#include <math.h>

#include "ws_device.cuh"

namespace ws {

enum { kModeAllReduce = 0, kModeLmHead = 1 };
constexpr int kFp8MaxRows = 8 * kConsumerWarps;  // activation rows of one launch of this kernel: eight per consumer warp

struct Fp8RankArgs {
    const void *x;
    const void *scales;
    float *out;        // all-reduce mode: [m, n]
    float *logits;     // lm_head mode: [m, vocab] or null
    uint32_t *argmax;  // lm_head mode: [m] or null
    int64_t ldx, scale_ld, row0, k0, vocab_row0;
    RankCtx ctx;
};

struct alignas(64) Fp8Params {
    // TMA descriptors first: the TMA unit fetches them from the parameter block, and they are
    // fetched fastest from its first bytes.  Per rank: weight shard [n rows][k bytes] as boxes of
    // 128 bytes x 16 rows ([0]) and x `gran` rows ([1]), 128B swizzle.
    CUtensorMap tmap[WS_MAX_WORLD][2];
    int32_t m, n, k, x_dtype, scale_kind, bn, bk;
    int32_t world, mode, vocab, mp, nstages, nslot_max, skb;
    int32_t gather_logits, ragged;   // ragged = 0: leftover tiles go whole to the first CTAs
    int32_t bk_shift, bn_shift;      // log2 of the scale block edges
    int32_t part_rows, gran;         // partial rows reserved per token; row granularity (1,2,4,8) of the ragged share
    int32_t stage_bytes, pad0;         // bytes of one weight stage: a whole number of 2 KB boxes (fp8_stage_boxes)
    uint64_t timeout_ns;
    SymLayout lay;
    Fp8RankArgs r[WS_MAX_WORLD];
};

struct Fp8Smem {  // byte offsets from the 1024-aligned base
    int32_t stages, q, sa, sw, red, part, bars, misc, total;
};

// Boxes (16 rows x 128 bytes) per stage: a tile's kbox boxes are cut into equal stages of at most
// kBoxesPerStage, so that no stage travels half empty (7168 columns = 56 boxes: four stages of 14
// instead of 16 + 16 + 16 + 8).
__host__ __device__ inline int fp8_stage_boxes(int kbox) {
    const int per_tile = (kbox + kBoxesPerStage - 1) / kBoxesPerStage;
    return (kbox + per_tile - 1) / per_tile;
}

__host__ __device__ inline Fp8Smem fp8_smem_layout(int nstages, int kbox, int mp, int nslot_max, int skb,
                                                   int m, int part_rows) {
    Fp8Smem s{};
    int o = 0;
    s.stages = o; o += nstages * fp8_stage_boxes(kbox) * kBoxBytes;
    s.q = o;      o += kbox * 4 * mp * 32;  // E4M3 bytes, [kb][tok][32]
    s.sa = o;     o += kbox * 4 * (mp > 8 ? mp : 8) * 4;
    s.sw = o;     o += ((nslot_max * skb * 4 + 15) / 16) * 16;
    s.red = o;    o += 2 * kConsumerWarps * 128 * 4;
    s.part = o;   o += ((m * part_rows * 4 + 15) / 16) * 16;
    s.bars = o;   o += 2 * kMaxStages * 8;
    s.misc = o;   o += 128;
    s.total = o;
    return s;
}

// Row schedule shared by host and device.  Whole tiles: CTA c owns tiles [c*Gm, (c+1)*Gm).
// Leftover rows [Gm*ncta*16, n), in units of `gran` rows: CTA c takes units [c*U/ncta, (c+1)*U/ncta)
// (ragged), or, when ragged is off, CTA c < Rg takes leftover tile c whole.
struct RowPlan {
    int Gm, lb, e0, e1;  // whole tiles per CTA; first leftover row; this CTA's extra rows [e0, e1)
};
__host__ __device__ inline RowPlan row_plan(int n, int ncta, int cta, int ragged, int gran) {
    RowPlan r{};
    const int G = n / kGroupRows;
    r.Gm = G / ncta;
    r.lb = r.Gm * ncta * kGroupRows;
    const int L = n - r.lb;
    if (ragged) {
        const int U = L / gran;
        r.e0 = r.lb + gran * (int)((int64_t)cta * U / ncta);
        r.e1 = r.lb + gran * (int)((int64_t)(cta + 1) * U / ncta);
    } else {
        r.e0 = r.lb + cta * kGroupRows;
        r.e1 = r.e0 + kGroupRows;
        if (r.e0 >= n) r.e0 = r.e1 = n;
    }
    return r;
}

__device__ __forceinline__ bool cand_better(float v, uint32_t i, float bv, uint32_t bi) {
    return v > bv || (v == bv && i < bi);
}

// What follows a CTA's finished rows, in both decode kernels: the output, the all-reduce exchange, or the
// lm_head's logits and argmax.  The CTA holds `count` row slots; row_of(i) is the global row of slot i
// (negative: none), value(tok, i) its finished sum.  Called by the CT consumer threads.
template <int CT, typename P, typename RowOf, typename Value>
__device__ __forceinline__ void fp8_finish(const P &p, const Fp8RankArgs &A, const RankCtx &X, uint32_t seq, int tid, int count,
                                           RowOf row_of, Value value) {
    constexpr int CW = CT / 32;
    const int cta = blockIdx.x, ncta = gridDim.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bank = seq & 1u;
    auto for_rows = [&](auto fn) {  // fn(tok, global row, slot)
        for (int j = tid; j < p.m * count; j += CT) {
            const int tok = j / count, i = j - tok * count, row = row_of(i);
            if (row >= 0) fn(tok, row, i);
        }
    };
    if (p.mode == kModeAllReduce && p.world == 1) {
        for_rows([&](int tok, int row, int i) { A.out[(size_t)tok * p.n + row] = value(tok, i); });
        return;
    }
    const int nflag = kMaxCtas + kMaxShared;
    const uint32_t *myflags = reinterpret_cast<const uint32_t *>(X.sym[X.rank] + p.lay.flags_off) +
                              (size_t)bank * p.world * nflag;

    if (p.mode == kModeAllReduce) {
        // every thread sends its rows' partials to all ranks as tagged words, then folds the same
        // rows in rank order as the ranks' words arrive: no barrier, fence or flag in between
        const size_t astride = (size_t)p.lay.max_m * p.lay.max_n;
        for (int pr = 0; pr < p.world; ++pr) {
            uint64_t *dst = reinterpret_cast<uint64_t *>(X.sym[pr] + p.lay.slota_off) + ((size_t)bank * p.world + X.rank) * astride;
            for_rows([&](int tok, int row, int i) { st_word_sys(dst + (size_t)tok * p.n + row, seq, value(tok, i)); });
        }
        const uint64_t *slots = reinterpret_cast<const uint64_t *>(X.sym[X.rank] + p.lay.slota_off) +
                                (size_t)bank * p.world * astride;
        for_rows([&](int tok, int row, int) {
            const size_t off = (size_t)tok * p.n + row;
            A.out[off] = fold_words(slots, astride, off, p.world, seq, p.timeout_ns, X.status, kStatTimeoutPeerA);
        });
        return;
    }

    // ---- lm_head: gather rows, publish candidates, final argmax
    const bool gathers = p.gather_logits && p.world > 1;
    if (gathers) {
        for (int pr = 0; pr < p.world; ++pr) {
            float *dst = reinterpret_cast<float *>(X.sym[pr] + p.lay.gather_off) +
                         (size_t)bank * p.lay.max_m * (size_t)p.lay.max_vocab;
            for_rows([&](int tok, int row, int i) { dst[(size_t)tok * p.lay.max_vocab + A.vocab_row0 + row] = value(tok, i); });
        }
    } else if (A.logits != nullptr) {  // a lone rank's rows are final where they are
        for_rows([&](int tok, int row, int i) { A.logits[(size_t)tok * p.vocab + A.vocab_row0 + row] = value(tok, i); });
    }
    for (int tok = warp; tok < p.m; tok += CW) {  // a warp per token
        float bv = -INFINITY;
        uint32_t bi = 0xFFFFFFFFu;
        for (int i = lane; i < count; i += 32) {
            if (row_of(i) < 0) continue;
            const float v = value(tok, i);
            const uint32_t idx = (uint32_t)(A.vocab_row0 + row_of(i));
            if (v > -INFINITY && cand_better(v, idx, bv, bi)) { bv = v; bi = idx; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (cand_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (lane < p.world) {
            uint64_t *dst = reinterpret_cast<uint64_t *>(X.sym[lane] + p.lay.pairs_off) +
                            (((size_t)bank * p.world + X.rank) * kMaxCtas + cta) * p.lay.max_m + tok;
            *dst = ((uint64_t)__float_as_uint(bv) << 32) | bi;
        }
    }
    consumer_bar_n<CT>();  // the st.release.sys below is cumulative over the stores this barrier ordered
    if (tid < p.world) {
        uint32_t *f = reinterpret_cast<uint32_t *>(X.sym[tid] + p.lay.flags_off) +
                      ((size_t)bank * p.world + X.rank) * nflag;
        st_release_sys(f + cta, seq);
    }
    const bool copies = gathers && A.logits != nullptr;
    if (!copies && cta != 0) return;
    // every CTA of every rank has published (its flag follows all of its stores)
    for (int i = tid; i < p.world * ncta; i += CT)
        wait_flag(myflags + (size_t)(i / ncta) * nflag + (i % ncta), seq, p.timeout_ns, X.status, kStatTimeoutGather);
    consumer_bar_n<CT>();
    if (copies) {
        const float *gl = reinterpret_cast<const float *>(X.sym[X.rank] + p.lay.gather_off) +
                          (size_t)bank * p.lay.max_m * (size_t)p.lay.max_vocab;
        const int64_t per = ((int64_t)p.vocab + ncta - 1) / ncta;
        const int64_t v0 = (int64_t)cta * per, v1 = min((int64_t)p.vocab, v0 + per);
        for (int tok = 0; tok < p.m; ++tok)
            for (int64_t v = v0 + tid; v < v1; v += CT)
                A.logits[(size_t)tok * p.vocab + v] = __ldcg(gl + (size_t)tok * p.lay.max_vocab + v);
    }
    if (cta == 0 && A.argmax != nullptr) {
        const uint64_t *pairs = reinterpret_cast<const uint64_t *>(X.sym[X.rank] + p.lay.pairs_off) +
                                (size_t)bank * p.world * kMaxCtas * p.lay.max_m;
        for (int tok = warp; tok < p.m; tok += CW) {
            float bv = -INFINITY;
            uint32_t bi = 0xFFFFFFFFu;
            for (int i = lane; i < p.world * ncta; i += 32) {
                const uint64_t pr = ld_volatile_u64(pairs + ((size_t)(i / ncta) * kMaxCtas + (i % ncta)) * p.lay.max_m + tok);
                const float v = __uint_as_float((uint32_t)(pr >> 32));
                const uint32_t idx = (uint32_t)pr;
                if (cand_better(v, idx, bv, bi)) { bv = v; bi = idx; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (cand_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
            }
            if (lane == 0) A.argmax[tok] = (bi == 0xFFFFFFFFu) ? 0u : bi;
        }
    }
}

__device__ __forceinline__ void fp8_rowpar_kernel_body(const Fp8Params &p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);

    constexpr int CW = kConsumerWarps, CT = kConsumerThreads;
    const int vr = blockIdx.y, cta = blockIdx.x, ncta = gridDim.x;
    const Fp8RankArgs &A = p.r[vr];
    const RankCtx &X = A.ctx;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int kbox = (p.k + 127) >> 7;
    const int kb32 = p.k >> 5;  // real 32-wide K blocks
    const RowPlan R = row_plan(p.n, ncta, cta, p.ragged, p.gran);
    // tiles of this CTA: Gm whole ones, then the extra rows cut at 16-row boundaries (so that a
    // tile never straddles a weight-scale block); tile t covers rows [trow(t), trow(t) + tcnt(t))
    const int xa = R.e0, xb = R.e1;
    const int xmid = min(xb, (xa / kGroupRows + 1) * kGroupRows);
    const int nx = xb > xa ? (xb > xmid ? 2 : 1) : 0;
    const int ntile = R.Gm + nx;
    auto trow = [&](int t) { return t < R.Gm ? (cta * R.Gm + t) * kGroupRows : (t == R.Gm ? xa : xmid); };
    auto tcnt = [&](int t) { return t < R.Gm ? kGroupRows : (t == R.Gm ? xmid - xa : xb - xmid); };
    // A tile of cnt rows is staged with a row pitch of tpad(cnt) (next power of two), so that a
    // stage always carries 16-32 KB: one box column = tpad rows x 128 bytes.
    auto tpad = [](int cnt) { return cnt > 8 ? 16 : cnt > 4 ? 8 : cnt > 2 ? 4 : cnt > 1 ? 2 : 1; };

    const Fp8Smem S = fp8_smem_layout(p.nstages, kbox, p.mp, p.nslot_max, p.skb, p.m, p.part_rows);
    uint8_t *q_s = smem + S.q;
    float *sa_s = reinterpret_cast<float *>(smem + S.sa);
    float *sw_s = reinterpret_cast<float *>(smem + S.sw);
    float *red_s = reinterpret_cast<float *>(smem + S.red);
    float *part_s = reinterpret_cast<float *>(smem + S.part);  // [tok][part_rows], tile t at t*16
    const uint32_t stage0 = smem_u32(smem + S.stages);
    const uint32_t full0 = smem_u32(smem + S.bars), empty0 = full0 + kMaxStages * 8;
    const int NS = p.nstages;

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full0 + s * 8, 1);
            mbar_init(empty0 + s * 8, CW);
        }
        mbar_fence_init();
    }
    __syncthreads();

    // Let the next kernel on the stream begin (it only prefetches weights until its own wait).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == CW) {
        // ------------------------------------------------------------ TMA producer warp
        RingPos rp;
        int item = 0;
        for (int t = 0; t < ntile; ++t) {
            const int r0 = trow(t), cnt = tcnt(t);
            const int pad = tpad(cnt), cols = p.stage_bytes / (pad * 128);  // box columns one stage holds
            for (int b0 = 0; b0 < kbox; b0 += cols) {
                const int nb = min(cols, kbox - b0);
                const int s = rp.s;
                if (item++ == NS) wait_predecessor();
                if (!mbar_wait(empty0 + s * 8, rp.ph ^ 1u, X.status)) return;  // a wait gave up: stop streaming
                if (lane == 0) mbar_arrive_expect_tx(full0 + s * 8, (uint32_t)(nb * cnt * 128));
                __syncwarp();
                for (int col = lane; col < nb; col += 32) {
                    const uint32_t dst = stage0 + s * p.stage_bytes + col * pad * 128;
                    if (cnt == kGroupRows) {  // a whole tile is one 16-row box, a ragged one is cnt/gran small boxes
                        tma_load_2d(dst, &p.tmap[vr][0], (b0 + col) * 128, r0, full0 + s * 8);
                    } else {
                        for (int done = 0; done < cnt; done += p.gran)
                            tma_load_2d(dst + done * 128, &p.tmap[vr][1], (b0 + col) * 128, r0 + done, full0 + s * 8);
                    }
                }
                rp.next(NS);
            }
        }
        return;
    }

    // ---------------------------------------------------------------- consumer warps
    // Everything below may read what the previous kernel on the stream wrote (activations, the
    // step sequence, exchange slots): wait for it.  The producer warp above streams weights,
    // which are static, and does not wait.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t seq = step_begin(X);
    // Prologue: weight scales of the rows this CTA touches (loads issued first, stored last, so
    // their latency overlaps the activation loads), then the activation quantisation.
    // q_s[kb][tok][32] holds E4M3 bytes, sa_s[kb][tok(sast)] the block scale 2^e.
    const int sast = p.mp > 8 ? p.mp : 8;  // tokens per K block in sa_s
    const int64_t kcol0 = A.k0 >> p.bk_shift;
    const int64_t srow_lo = (A.row0 + (int64_t)cta * R.Gm * kGroupRows) >> p.bn_shift;
    const int nslotA = R.Gm ? (int)(((A.row0 + (int64_t)(cta + 1) * R.Gm * kGroupRows - 1) >> p.bn_shift) - srow_lo + 1) : 0;
    auto slot_of = [&](int t) {
        return t < R.Gm ? (int)(((A.row0 + (int64_t)trow(t)) >> p.bn_shift) - srow_lo) : nslotA + (t - R.Gm);
    };
    {
        const int ncols = (int)(((A.k0 + p.k - 1) >> p.bk_shift) - kcol0 + 1);
        const int nsw = (nslotA + nx) * ncols;
        auto load_scale = [&](int i) -> float {
            const int sl = i / ncols, c = i - sl * ncols;
            const int64_t srow = sl < nslotA ? srow_lo + sl : (A.row0 + (int64_t)trow(R.Gm + sl - nslotA)) >> p.bn_shift;
            const int64_t idx = srow * A.scale_ld + kcol0 + c;
            if (p.scale_kind == WS_SCALE_UE8M0) {
                const uint32_t b = __ldg(static_cast<const uint8_t *>(A.scales) + idx);
                return (b == 0xFFu) ? __uint_as_float(0x7FC00000u)
                                    : (b == 0u ? __uint_as_float(0x00400000u) : __uint_as_float(b << 23));
            }
            return __ldg(static_cast<const float *>(A.scales) + idx);
        };
        auto sw_index = [&](int i) { return (i / ncols) * p.skb + (i - (i / ncols) * ncols); };
        float pre[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = tid + u * CT;
            pre[u] = i < nsw ? load_scale(i) : 0.0f;
        }
        for (int i = tid; i < kbox * 4 * sast; i += CT)  // tokens the launch does not carry
            if ((i % sast) >= p.m) sa_s[i] = 0.0f;
        const int chunks_per_row = kbox * 16;  // 8-element chunks over the padded K
        const int total = p.mp * chunks_per_row;
        // four chunks per thread and pass: all loads are in flight before the first is used
        for (int c0 = tid; c0 < ((total + 31) & ~31); c0 += 4 * CT) {
            float v[4][8];
            int tok[4], ch[4];
            bool valid[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + u * CT;
                tok[u] = p.mp == 1 ? 0 : c / chunks_per_row;
                ch[u] = c - tok[u] * chunks_per_row;
                valid[u] = (c < total) && (tok[u] < p.m) && (ch[u] * 8 < p.k);
                load_act8(A.x, p.x_dtype, (int64_t)tok[u] * A.ldx + ch[u] * 8, valid[u], v[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + u * CT;
                if (c >= ((total + 31) & ~31)) break;  // warp-uniform
                int e;
                uint32_t lo, hi;
                act_quant8(v[u], e, lo, hi);
                if (c < total) {
                    const int kb = ch[u] >> 2;
                    *reinterpret_cast<uint2 *>(q_s + ((size_t)(kb * p.mp + tok[u]) * 32 + (ch[u] & 3) * 8)) =
                        valid[u] ? make_uint2(lo, hi) : make_uint2(0u, 0u);
                    if ((ch[u] & 3) == 0) sa_s[kb * sast + tok[u]] = valid[u] ? pow2_f32(e) : 0.0f;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = tid + u * CT;
            if (i < nsw) sw_s[sw_index(i)] = pre[u];
        }
        for (int i = tid + 4 * CT; i < nsw; i += CT) sw_s[sw_index(i)] = load_scale(i);
    }
    consumer_bar_n<CT>();

    const int g = lane >> 2, tq = lane & 3;
    const int lm_row = (lane & 7) + ((lane >> 3) & 1) * 8;  // ldmatrix source row of this lane
    const int lm_hi = lane >> 4;                            // 0: k 0..15 of the block, 1: k 16..31
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    RingPos rp;
    int redbuf = 0;

    const int kofs = (int)(A.k0 - kcol0 * p.bk);  // k0 modulo the scale block
    // shared-space addresses of this lane's operands of K block 0 (advanced per block below)
    // More than eight activation rows ("wide"): warp w takes rows 8w..8w+7 of the activations
    // (MMA columns) for every box of a tile, so each warp owns a 16 x 8 block of the output and
    // nothing is combined across warps; the weights are staged once for all rows.
    const bool wide = p.mp > 8;
    const int tg = wide ? warp : 0;                 // this warp's group of eight activation rows
    const bool tg_active = !wide || tg * 8 < p.mp;
    const uint32_t q_lane = smem_u32(q_s) + (uint32_t)((tg * 8 + g) * 32 + tq * 4);
    const uint32_t q_step = (uint32_t)(p.mp * 32);
    const uint32_t sa_lane = smem_u32(sa_s) + (uint32_t)((tg * 8 + tq * 2) * 4);
    const uint32_t sa_step = (uint32_t)(sast * 4);
    const bool has_b = tg * 8 + g < p.mp;
    auto mma_step = [&](uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, int kb, uint32_t swrow) {
        uint32_t b0r = 0, b1r = 0;
        if (has_b) {
            b0r = lds_u32(q_lane + kb * q_step);
            b1r = lds_u32(q_lane + kb * q_step + 16);
        }
        float d[4];
        mma_e4m3_16x8x32(d, a0, a1, a2, a3, b0r, b1r);
        const float2 sa = lds_f32x2(sa_lane + kb * sa_step);
        const float sw = lds_f32(swrow + (uint32_t)(((kofs + kb * 32) >> p.bk_shift) * 4));
        const float f0 = sa.x * sw, f1 = sa.y * sw;
        acc[0] = fmaf(d[0], f0, acc[0]);
        acc[1] = fmaf(d[1], f1, acc[1]);
        acc[2] = fmaf(d[2], f0, acc[2]);
        acc[3] = fmaf(d[3], f1, acc[3]);
    };
    auto run_item = [&](int b0, int nb, int slot, int pad) {
        const int s = rp.s;
        const bool landed = mbar_wait(full0 + s * 8, rp.ph, X.status);  // false: a wait gave up, the step is void
        const uint32_t sbase = stage0 + s * p.stage_bytes;
        const uint32_t swrow = smem_u32(sw_s) + (uint32_t)(slot * p.skb * 4);
        for (int bi = wide ? 0 : warp; bi < nb && tg_active && landed; bi += wide ? 1 : CW) {
            const int box = b0 + bi;
            const uint32_t bbase = sbase + bi * pad * 128 + lm_row * 128;
            const uint32_t sw7 = (uint32_t)((bi * pad + lm_row) & 7);  // 128B-swizzle phase of this row's address
            if (box * 4 + 4 <= kb32) {  // full box: issue the four fragment loads together
                uint32_t a[4][4];
#pragma unroll
                for (int kq = 0; kq < 4; ++kq)
                    ldmatrix_x4(bbase + ((((uint32_t)(kq << 1) | lm_hi) ^ sw7) << 4), a[kq][0], a[kq][1], a[kq][2], a[kq][3]);
#pragma unroll
                for (int kq = 0; kq < 4; ++kq) mma_step(a[kq][0], a[kq][1], a[kq][2], a[kq][3], box * 4 + kq, swrow);
            } else {
                for (int kq = 0; kq < 4 && box * 4 + kq < kb32; ++kq) {
                    uint32_t a0, a1, a2, a3;
                    ldmatrix_x4(bbase + ((((uint32_t)(kq << 1) | lm_hi) ^ sw7) << 4), a0, a1, a2, a3);
                    mma_step(a0, a1, a2, a3, box * 4 + kq, swrow);
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + s * 8);
        rp.next(NS);
    };
    // Sum the consumer warps' accumulators in warp order; thread t < 128 ends with
    // the value of (row = t & 15, tok = t >> 4).
    auto reduce_warps = [&]() -> float {
        float *rb = red_s + (redbuf * CW + warp) * 128;
        rb[(2 * tq) * 16 + g] = acc[0];
        rb[(2 * tq + 1) * 16 + g] = acc[1];
        rb[(2 * tq) * 16 + g + 8] = acc[2];
        rb[(2 * tq + 1) * 16 + g + 8] = acc[3];
        consumer_bar_n<CT>();
        float v = 0.0f;
        if (tid < 128) {
            const float *r0 = red_s + redbuf * CW * 128 + tid;
            v = r0[0];
#pragma unroll
            for (int w = 1; w < CW; ++w) v += r0[w * 128];
        }
        redbuf ^= 1;
        return v;
    };

    const int row_t = tid & 15, tok_t = tid >> 4;  // meaningful for tid < 128
    const int PR = p.part_rows;

    for (int t = 0; t < ntile; ++t) {
        const int slot = slot_of(t);
        const int pad = tpad(tcnt(t)), cols = p.stage_bytes / (pad * 128);
        acc[0] = acc[1] = acc[2] = acc[3] = 0.0f;
        for (int b0 = 0; b0 < kbox; b0 += cols) run_item(b0, min(cols, kbox - b0), slot, pad);
        if (wide) {  // the accumulator fragment is final: rows g, g + 8 x tokens 8 tg + 2 tq, + 1
            const int tk0 = tg * 8 + 2 * tq;
            if (tk0 < p.m) {
                part_s[tk0 * PR + t * kGroupRows + g] = acc[0];
                part_s[tk0 * PR + t * kGroupRows + g + 8] = acc[2];
            }
            if (tk0 + 1 < p.m) {
                part_s[(tk0 + 1) * PR + t * kGroupRows + g] = acc[1];
                part_s[(tk0 + 1) * PR + t * kGroupRows + g + 8] = acc[3];
            }
            continue;
        }
        const float v = reduce_warps();
        if (tid < 128 && tok_t < p.m) part_s[tok_t * PR + t * kGroupRows + row_t] = v;
    }
    consumer_bar_n<CT>();  // part_s complete

    fp8_finish<CT>(p, A, X, seq, tid, ntile * kGroupRows,
                   [&](int i) { const int t = i >> 4, r = i & 15; return r < tcnt(t) ? trow(t) + r : -1; },
                   [&](int tok, int i) { return part_s[tok * PR + i]; });
}

__global__ void __launch_bounds__(kThreads, 1) fp8_rowpar_kernel(const __grid_constant__ Fp8Params p) {
    const RankCtx &X = p.r[blockIdx.y].ctx;
    fp8_rowpar_kernel_body(p);
    if (p.world > 1 || p.mode == kModeLmHead) {  // a lone all-reduce rank exchanges nothing
        // step_begin again: the value is unchanged until the last CTA publishes the next one below
        step_end(X, step_begin(X), gridDim.x);
    }
    host_done_signal(X, gridDim.x);
}

}  // namespace ws

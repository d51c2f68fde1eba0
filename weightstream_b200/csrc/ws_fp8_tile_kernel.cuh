// FP8 E4M3 GEMM of many activation rows (prefill) on the 5th-generation tensor cores with block scaling
// (sm_100a), one launch for all of them: the output is cut into tiles of 128 weight rows x up to 224 tokens
// and persistent CTAs take tiles in turn, token tiles fastest, so that the CTAs of a wave share weight rows
// in L2.  The decode kernel (ws_fp8_bs_kernel.cuh) keeps a CTA's rows and streams all K once for at most
// 128 tokens; looping it over 2000 tokens read the weights 16 times and was bound by its read-back.
//
// Per 128-wide K slab a stage holds the tile's weight rows (TMA box, 128B swizzle), the token tile's
// quantised activations and their scale atoms (one bulk copy; layout of act_prep_kernel).  Warp 0 feeds the
// ring, warp 1 issues four MMAs per slab (M = 128, N = tokens).  fp32 weight scales: every slab goes to one of
// two accumulators, and the two epilogue warpgroups (one half of the tokens each) read it back and add it x
// the scale to registers while the next slab's MMAs fill the other; the register file is split by
// setmaxnreg, 112 sums per thread do not fit an even share.  UE8M0 weight scales (WUE) are an MMA operand,
// whose atoms warps 2 and 3 lay out; an accumulator takes two slabs (see bs_chain).
//
// Bound: with fp32 scales the hand-off and read-back of an accumulator per slab (2000 rows of K 8192 150 us a step, and no
// faster without the activation loads; 9.7 TB/s out of L2, tensor pipe 41 %); with UE8M0 scales, half the read-backs, what
// L2 hands the SMs (131 us, 12 TB/s).  Wide token tiles favour both: 16 KB + 128 bytes per token a slab.
#pragma once

#include "ws_fp8_bs_kernel.cuh"

namespace ws {

constexpr int kTileTokens = 224;   // most tokens of a tile: two accumulators and the scale columns fill tensor memory
constexpr int kTileThreads = 384;  // warpgroup 0: producer, MMA issue, scale atoms (UE8M0); 1 and 2: epilogue
constexpr int kTileMaxStages = 8;
constexpr int kTileRegsFeed = 56, kTileRegsSum = 216;  // registers a thread of warpgroup 0 / of 1 and 2: 128 x 56 + 256 x 216 <= 384 x 168

struct alignas(64) TileParams {
    CUtensorMap tmap_w;                // weight shard [n][k bytes], box 128 bytes x 128 rows, 128B swizzle
    const uint8_t *xq;                 // [token tile][ks][8 chunks][tokens][16] + atoms: see act_prep_kernel
    const void *scales;
    float *out;
    int64_t scale_ld, row0, k0;
    int32_t m, n, k, ks, bn_shift, bk_shift;
    int32_t tokens, ntok, nrow;        // tokens per tile; token and row tiles
    int32_t nstages, x_pitch;
    RankCtx ctx;
};

struct TileSmem {
    int32_t a, x, wsf, bars, misc, total;
};
__host__ __device__ inline TileSmem tile_smem_layout(int nstages, int x_pitch, bool wue) {
    TileSmem s{};
    int o = 0;
    s.a = o;    o += nstages * 16384;
    s.x = o;    o += nstages * x_pitch + 4096;  // (columns past a tile's tokens read up to 224 x 16 bytes on)
    s.wsf = o;  o += (wue ? nstages : 1) * kBsAtomBytes;
    s.bars = o; o += (2 * kTileMaxStages + 4) * 8;
    s.misc = o; o += 16;
    s.total = o;
    return s;
}

// The first `nc` columns of an accumulator, times the weight scale (SCALED), added to a thread's sums; C columns per
// round trip to tensor memory.
template <int C, bool SCALED>
__device__ __forceinline__ void read_back(float (&acc)[kTileTokens / 2], uint32_t t, int nc, float sw) {
    constexpr int CP = kTileTokens / 2;
#pragma unroll
    for (int c = 0; c < CP; c += C) {
        if (c < nc) {  // warp-uniform
            if (c + C <= CP) {
                uint32_t r[C];
                tmem_ld_cols<C>(t + (uint32_t)c, r);
#pragma unroll
                for (int i = 0; i < C; ++i) acc[c + i] = SCALED ? fmaf(__uint_as_float(r[i]), sw, acc[c + i]) : acc[c + i] + __uint_as_float(r[i]);
            } else {
                uint32_t r[16];
                tmem_ld_cols<16>(t + (uint32_t)c, r);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[c + i] = SCALED ? fmaf(__uint_as_float(r[i]), sw, acc[c + i]) : acc[c + i] + __uint_as_float(r[i]);
            }
        }
    }
}

template <bool WUE>
__global__ void __launch_bounds__(kTileThreads, 1) fp8_tile_kernel(const __grid_constant__ TileParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
    const int NS = p.nstages, KS = p.ks, ntiles = p.nrow * p.ntok;
    const TileSmem S = tile_smem_layout(NS, p.x_pitch, WUE);
    const uint32_t a0 = smem_u32(smem + S.a), x0 = smem_u32(smem + S.x), wsf0 = smem_u32(smem + S.wsf);
    // full[s]: the stage's bytes landed (and its scale atom is laid out); done[s]: its MMAs have completed (stage
    // free; the last of an accumulator's: accumulator ready); accempty[g]: accumulator g has been read
    const uint32_t full0 = smem_u32(smem + S.bars), done0 = full0 + kTileMaxStages * 8;
    const uint32_t accempty0 = done0 + kTileMaxStages * 8;
    constexpr int EW = 8, CH = bs_chain(WUE);
    uint32_t *const status = p.ctx.status;
    if (warp == 0) {
        if (elect_one()) {
            for (int s = 0; s < NS; ++s) {
                mbar_init(full0 + s * 8, WUE ? 3 : 1);
                mbar_init(done0 + s * 8, 1);
            }
            // (two are used; with two initialised, fp32 scales took 155 us for 2000 rows of K 8192 instead of 150, in
            // every form of the loops below that was tried: how the CTAs of a wave meet in L2 depends on their start)
            for (int g = 0; g < 4; ++g) mbar_init(accempty0 + g * 8, g < 2 ? EW : 1);
            mbar_fence_init();
        }
        __syncwarp();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(smem + S.misc), 512);
        tmem_relinquish();
    }
    if (!WUE && tid >= 256) {
        reinterpret_cast<uint32_t *>(smem + S.wsf)[tid - 256] = 0x7F7F7F7Fu;  // the weight operand's scale: 2^0
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + S.misc);
    const uint32_t t_sf = tmem + 2u * kTileTokens, t_sfa = t_sf + 16u;  // two sets of 8 activation-scale columns, then the weights'
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int atom = bs_atom_bytes(p.tokens);  // (of a full tile; the last tile's may be smaller)
    const int64_t tile_bytes = (int64_t)KS * (p.tokens * 128 + atom);

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTileRegsFeed));
        if (warp == 0) {
            // -------------------------------------------------------- producer (one thread)
            if (elect_one()) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                int s = 0, lap = 0;
                uint32_t ph = 1;
                bool ok = true;
                for (int q = blockIdx.x; q < ntiles && ok; q += gridDim.x) {
                    const int rt = q / p.ntok, tt = q - rt * p.ntok, mt = min(p.tokens, p.m - tt * p.tokens);
                    const uint32_t x_slab = (uint32_t)(mt * 128 + bs_atom_bytes(mt));
                    const uint8_t *xq = p.xq + (int64_t)tt * tile_bytes;
                    for (int k = 0; k < KS; ++k, xq += x_slab) {
                        if (lap > 0 && !mbar_wait(done0 + s * 8, ph, status)) { ok = false; break; }
                        mbar_arrive_expect_tx(full0 + s * 8, 16384u + x_slab);
                        tma_load_2d(a0 + s * 16384, &p.tmap_w, k * 128, rt * 128, full0 + s * 8);
                        bulk_load(x0 + s * p.x_pitch, xq, x_slab, full0 + s * 8);
                        if (++s == NS) { s = 0; ++lap; ph ^= 1u; }
                    }
                }
            }
        } else if (warp == 1) {
            // -------------------------------------------------------- MMA issue (one thread)
            if (elect_one()) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                if (!WUE) tmem_cp_atom(t_sfa, umma_desc(wsf0, 128, false));
                const uint32_t a_lo0 = umma_desc_lo(a0), x_lo0 = (x0 & 0x3FFFFu) >> 4, x_stage = (uint32_t)p.x_pitch >> 4;
                const uint64_t sf0 = umma_desc(x0, 128, false), wsf_d0 = umma_desc(wsf0, 128, false);
                int s = 0;
                uint32_t ph = 0, g = 0, acc_ph = 1, odd = 0;
                bool ok = true;
                for (int q = blockIdx.x; q < ntiles && ok; q += gridDim.x) {
                    const int tt = q % p.ntok, mt = min(p.tokens, p.m - tt * p.tokens);
                    const uint32_t m16 = (uint32_t)mt, x_kb = 2u * m16;
                    const int cols = (mt + 15) / 16 * 16;
                    uint32_t id[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) id[j] = bs_idesc(cols, WUE ? j : 0, j);
                    for (int k = 0; k < KS; ++k) {
                        if (k % CH == 0 && !mbar_wait(accempty0 + g * 8, acc_ph, status)) { ok = false; break; }
                        if (!mbar_wait(full0 + s * 8, ph, status)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t a = a_lo0 + (uint32_t)s * 1024u, x_off = (uint32_t)s * x_stage, b = (x_lo0 + x_off) | (m16 << 16);
                        const uint32_t d = tmem + g * kTileTokens, sx = t_sf + odd * 8u, sw = WUE ? t_sfa + odd * 4u : t_sfa;
                        const uint64_t sf = sf0 + (uint64_t)(x_off + 8u * m16);
                        tmem_cp_atom(sx, sf);
                        if (mt > 128) tmem_cp_atom(sx + 4, sf + 32);
                        if (WUE) tmem_cp_atom(sw, wsf_d0 + (uint64_t)((uint32_t)s * (kBsAtomBytes >> 4)));
                        umma_bs_ss(d, a, b, kUmmaDescHiSw128, kUmmaDescHiX, id[0], sw, sx, k % CH ? 1u : 0u);
                        umma_bs_ss(d, a + 2, b + x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id[1], sw, sx, 1u);
                        umma_bs_ss(d, a + 4, b + 2 * x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id[2], sw, sx, 1u);
                        umma_bs_ss(d, a + 6, b + 3 * x_kb, kUmmaDescHiSw128, kUmmaDescHiX, id[3], sw, sx, 1u);
                        umma_commit(done0 + s * 8);
                        odd ^= 1u;
                        if (++s == NS) { s = 0; ph ^= 1u; }
                        if (k % CH == CH - 1 || k == KS - 1) {
                            g ^= 1u;
                            if (g == 0) acc_ph ^= 1u;
                        }
                    }
                }
            }
        } else if constexpr (WUE) {
            // -------------------------------------------------------- scale atoms (thread = rows r and r + 64)
            const int r = tid - 64;
            const Ue8m0Scales sc(p.scales, p.scale_ld, p.k0, p.k, p.bk_shift);
            int s = 0, lap = 0, lq = blockIdx.x, lk = 0;  // stage to fill; tile and slab to load
            uint32_t ph = 1;
            const uint8_t *row_lo = nullptr, *row_hi = nullptr;
            auto load = [&](uint32_t (&w)[2]) {
                if (lq >= ntiles) return false;
                if (lk == 0) {
                    const int row = lq / p.ntok * 128 + r;
                    row_lo = sc.row((p.row0 + min(row, p.n - 1)) >> p.bn_shift);
                    row_hi = sc.row((p.row0 + min(row + 64, p.n - 1)) >> p.bn_shift);
                }
                w[0] = sc.slab(row_lo, lk);
                w[1] = sc.slab(row_hi, lk);
                if (++lk == KS) { lk = 0; lq += gridDim.x; }
                return true;
            };
            const uint32_t at = wsf0 + (uint32_t)((r & 31) * 16 + (r >> 5) * 4);
            auto put = [&](const uint32_t (&w)[2], bool ok) {
                if (lap == 1 && s == 0) wait_predecessor();
                if (ok && lap > 0) ok = mbar_wait(done0 + s * 8, ph, status);
                if (!__all_sync(0xffffffffu, ok)) return false;
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + s * kBsAtomBytes), "r"(w[0]) : "memory");
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + s * kBsAtomBytes + 8), "r"(w[1]) : "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + s * 8);
                if (++s == NS) { s = 0; ++lap; ph ^= 1u; }
                return true;
            };
            uint32_t w0[2], w1[2], w2[2];  // three slabs' words in flight
            bool h0 = load(w0), h1 = load(w1), h2 = load(w2);
            for (;;) {
                if (!put(w0, h0)) break;
                h0 = load(w0);
                if (!put(w1, h1)) break;
                h1 = load(w1);
                if (!put(w2, h2)) break;
                h2 = load(w2);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue warps
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTileRegsSum));
        const int quad = warp & 3, rc = quad * 32 + lane, half = (warp >> 2) - 1;  // TMEM lane quarter; which half of the tokens
        const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16);
        asm volatile("griddepcontrol.wait;" ::: "memory");
        constexpr int CP = kTileTokens / 2;
        const int hcols = (p.tokens / 2 + 15) / 16 * 16;  // columns of the first half: whole groups of 16
        const int64_t kcol0 = p.k0 >> p.bk_shift;
        const int kofs = (int)(p.k0 - (kcol0 << p.bk_shift));
        int s = 0;
        uint32_t ph = 0, g = 0;
        bool ok = true;
        for (int q = blockIdx.x; q < ntiles; q += gridDim.x) {
            const int rt = q / p.ntok, tt = q - rt * p.ntok, mt = min(p.tokens, p.m - tt * p.tokens);
            const int c0 = half * hcols, nc = min(mt - c0, half == 0 ? hcols : CP);  // this half's columns (may be none)
            const int row = rt * 128 + rc;
            float acc[CP];
#pragma unroll
            for (int i = 0; i < CP; ++i) acc[i] = 0.0f;
            if constexpr (WUE) {
                for (int k = 0; k < KS; k += CH) {
                    s += min(CH, KS - k) - 1;  // the accumulator's last slab
                    if (s >= NS) { s -= NS; ph ^= 1u; }
                    if (ok && !mbar_wait_inline(done0 + s * 8, ph, status)) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                    tc_fence_after();
                    if (ok) read_back<16, false>(acc, tl + g * kTileTokens + (uint32_t)c0, nc, 1.0f);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accempty0 + g * 8);
                    g ^= 1u;
                    if (++s == NS) { s = 0; ph ^= 1u; }
                }
            } else {
                const float *sw_row = static_cast<const float *>(p.scales) + ((p.row0 + min(row, p.n - 1)) >> p.bn_shift) * p.scale_ld + kcol0;
                float sw = __ldg(sw_row + (kofs >> p.bk_shift));
                for (int k = 0; k < KS; ++k) {
                    const float next = k + 1 < KS ? __ldg(sw_row + ((kofs + (k + 1) * 128) >> p.bk_shift)) : 0.0f;
                    if (ok && !mbar_wait_inline(done0 + s * 8, ph, status)) ok = false;  // (no call: it would not leave the sums their registers)
                    ok = __all_sync(0xffffffffu, ok);
                    tc_fence_after();
                    if (ok) read_back<32, true>(acc, tl + g * kTileTokens + (uint32_t)c0, nc, sw);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accempty0 + g * 8);
                    g ^= 1u;
                    if (++s == NS) { s = 0; ph ^= 1u; }
                    sw = next;
                }
            }
            if (row < p.n) {
                int64_t ld = p.n;
                asm volatile("" : "+l"(ld));  // offsets computed here, not kept in registers through the loop
                float *dst = p.out + ((int64_t)tt * p.tokens + c0) * ld + row;
#pragma unroll
                for (int i = 0; i < CP; ++i) {
                    if (i < nc) *dst = acc[i];
                    dst += ld;
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    host_done_signal(p.ctx, gridDim.x);
}

}  // namespace ws

// FP8 E4M3 row-parallel decode step for one or two activation rows on CUDA cores, fused with its
// exchange (sm_100a).  One persistent CTA per SM (two where they fit: the next step's CTA then fills its
// ring while this one finishes).
//
// A CTA owns a contiguous range of output rows, floor or ceil of n / ncta, so all SMs stream the same
// bytes to within a row.  One producer warp brings whole rows in by bulk copy, R rows per stage.  The
// eight consumer warps are S slices of K times G row groups; a lane owns the same C 16-byte chunks of K
// in every row its warp visits, and holds that K's activations in registers as f16 pairs: it quantises
// them itself, straight from memory, exactly as the reference does
// (crates/weightstream-ref/src/actquant.rs:21-57), so no shared memory, barrier or other warp stands
// between the predecessor's end and the first product.  Per row and chunk: one conflict-free 128-bit
// shared load, 8 conversions to f16 pairs, 16 mixed-precision FMAs with exact products
// (fma.rn.f32.f16), one FMA with the product of the block scales; four rows are in flight at a time and
// their sums are folded over the lanes by six shuffles.  Slices meet once, after the last row, in slice order.
//
// Bound: HBM for large shards, the dependency latency between steps for small ones.
#pragma once

#include <math.h>

#include "ws_device.cuh"
#include "ws_fp8_kernel.cuh"

namespace ws {

constexpr int kGemvMaxSlices = kConsumerWarps;

struct alignas(64) Fp8GemvParams {
    int32_t m, n, k, x_dtype, scale_kind, world, mode, vocab;
    int32_t bk_shift, bn_shift, nslot_max, skb;
    int32_t slices, rows_per_stage, nstages, rows_max, stage_bytes, gather_logits;
    int32_t ahead;  // groups of warps (0 or 1) that ask for the activations ahead of the wait on the predecessor
    uint64_t timeout_ns;
    SymLayout lay;
    Fp8RankArgs r[WS_MAX_WORLD];
    const uint8_t *w[WS_MAX_WORLD];
    int64_t ldw[WS_MAX_WORLD];
};

struct Fp8GemvSmem {
    int32_t stages, sw, part, bars, total;
};
__host__ __device__ inline Fp8GemvSmem fp8_gemv_smem(int nstages, int stage_bytes, int nslot_max, int skb, int m, int slices, int rows_max) {
    Fp8GemvSmem s{};
    int o = 0;
    s.stages = o; o += nstages * stage_bytes;
    s.sw = o;     o += (nslot_max * skb * 4 + 15) / 16 * 16;
    s.part = o;   o += (m * slices * rows_max * 4 + 15) / 16 * 16;  // [token][slice][row of the CTA]
    s.bars = o;   o += 2 * kMaxStages * 8;
    s.total = o;
    return s;
}

template <int GT, int C>
__device__ __forceinline__ void fp8_gemv_body(const Fp8GemvParams &p) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int CW = kConsumerWarps, CT = kConsumerThreads;
    const int vr = blockIdx.y, cta = blockIdx.x, ncta = gridDim.x;
    const Fp8RankArgs &A = p.r[vr];
    const RankCtx &X = A.ctx;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row_a = (int)((int64_t)p.n * cta / ncta), rows = (int)((int64_t)p.n * (cta + 1) / ncta) - row_a;
    const int R = p.rows_per_stage, NS = p.nstages, items = (rows + R - 1) / R;

    const Fp8GemvSmem L = fp8_gemv_smem(NS, p.stage_bytes, p.nslot_max, p.skb, GT, p.slices, p.rows_max);
    float *sw_s = reinterpret_cast<float *>(smem + L.sw), *part_s = reinterpret_cast<float *>(smem + L.part);
    const uint32_t stage0 = smem_u32(smem + L.stages);
    const uint32_t full0 = smem_u32(smem + L.bars), empty0 = full0 + kMaxStages * 8;
    if (tid == CT) {  // the producer's first lane
        for (int s = 0; s < NS; ++s) {
            mbar_init(full0 + s * 8, 1);
            mbar_init(empty0 + s * 8, CW);
        }
        mbar_fence_init();
    }
    __syncthreads();
    // Let the next kernel on the stream begin (it only streams weights until its own wait).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == CW) {
        // ------------------------------------------------------------ producer warp
        const uint8_t *w = p.w[vr] + (int64_t)row_a * p.ldw[vr];
        const bool dense = p.ldw[vr] == p.k;
        RingPos rp;
        for (int it = 0; it < items; ++it, rp.next(NS)) {
            const int s = rp.s, r0 = it * R, nr = min(R, rows - r0);
            if (it == NS) wait_predecessor();
            if (!mbar_wait(empty0 + s * 8, rp.ph ^ 1u, X.status)) return;  // a wait gave up: stop streaming
            if (lane == 0) mbar_arrive_expect_tx(full0 + s * 8, (uint32_t)(nr * p.k));
            __syncwarp();
            const uint32_t dst = stage0 + s * p.stage_bytes;
            if (dense ? lane == 0 : lane < nr)  // adjacent rows of a dense shard are one copy
                bulk_load(dst + lane * p.k, w + (int64_t)(r0 + lane) * p.ldw[vr], (uint32_t)(dense ? nr * p.k : p.k), full0 + s * 8);
        }
        return;
    }

    // ---------------------------------------------------------------- consumer warps
    const int S = p.slices, G = CW / S;
    const int slice = warp % S, grp = warp / S;  // warps beyond S * G only keep the barriers moving
    const int64_t kcol0 = A.k0 >> p.bk_shift, srow_lo = (A.row0 + row_a) >> p.bn_shift;
    {   // weight scales of this CTA's rows: static, so fetched before the wait on the predecessor
        const int ncols = (int)(((A.k0 + p.k - 1) >> p.bk_shift) - kcol0 + 1);
        const int nslot = rows > 0 ? (int)(((A.row0 + row_a + rows - 1) >> p.bn_shift) - srow_lo + 1) : 0;
        for (int i = tid; i < nslot * ncols; i += CT) {
            const int sl = i / ncols, c = i - sl * ncols;
            const int64_t idx = (srow_lo + sl) * A.scale_ld + kcol0 + c;
            float v;
            if (p.scale_kind == WS_SCALE_UE8M0) v = e8m0_f32(__ldg(static_cast<const uint8_t *>(A.scales) + idx));
            else v = __ldg(static_cast<const float *>(A.scales) + idx);
            sw_s[sl * p.skb + c] = v;
        }
    }
    // One warp of each slice of K asks for its activations.  (All warps asking, 148 CTAs of them, queued at the few lines
    // that a small K is: two rows of 7168 x 512 4.8 us a step without, 5.9 with all eight, 4.6 with one; of 1024 x 512 3.7,
    // 4.7, 3.5; of K 2048 and up, no difference.  A branch around the loop instead of a test in it: 8 virtual ranks, one row
    // of K 8192, which ask for nothing, 26.8 us, 25.8 so.)
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int k = ((slice * C + i) * 32 + lane) * 16;
        if (k < p.k && grp < p.ahead)
#pragma unroll
            for (int t = 0; t < GT; ++t) prefetch_act(A.x, p.x_dtype, (int64_t)t * A.ldx + k);
    }
    consumer_bar();
    // Everything below may read what the previous kernel on the stream wrote (activations, the step
    // sequence, exchange slots).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint32_t xh[GT][C][8];  // this lane's quantised activations
    float sa[GT][C];        // and their block scales 2^e
    int swc[C];             // column of each chunk in sw_s
    bool live[C];
    {
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const int k = ((slice * C + i) * 32 + lane) * 16;
            live[i] = k < p.k && grp < G;
            swc[i] = live[i] ? (int)(((A.k0 + k) >> p.bk_shift) - kcol0) : 0;
        }
        float v[GT][C][16];
#pragma unroll
        for (int t = 0; t < GT; ++t)
#pragma unroll
            for (int i = 0; i < C; ++i) {
                const int k = ((slice * C + i) * 32 + lane) * 16;
                load_act8(A.x, p.x_dtype, (int64_t)t * A.ldx + k, live[i], *reinterpret_cast<float(*)[8]>(v[t][i]));
                load_act8(A.x, p.x_dtype, (int64_t)t * A.ldx + k + 8, live[i], *reinterpret_cast<float(*)[8]>(v[t][i] + 8));
            }
#pragma unroll
        for (int t = 0; t < GT; ++t)
#pragma unroll
            for (int i = 0; i < C; ++i) {
                int e;
                const uint4 q = act_quant16(v[t][i], e);  // a 32-block is two adjacent lanes
                const uint32_t qq[4] = {q.x, q.y, q.z, q.w};
                sa[t][i] = live[i] ? pow2_f32(e) : 0.0f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    xh[t][i][2 * j] = live[i] ? e4m3x2_half_to_f16x2<0>(qq[j]) : 0u;
                    xh[t][i][2 * j + 1] = live[i] ? e4m3x2_half_to_f16x2<1>(qq[j]) : 0u;
                }
            }
    }
    const bool solo = p.mode == kModeAllReduce && p.world == 1;
    const uint32_t seq = solo ? 0u : step_begin(X);

    // byte offset of each chunk inside a row; lanes past the end of K read the row's first chunk and multiply
    // it by zero activations and a zero factor (a NaN weight there is in the row's sum anyway; an infinite scale
    // must not become one)
    uint32_t off[C];
#pragma unroll
    for (int i = 0; i < C; ++i) off[i] = live[i] ? (uint32_t)(((slice * C + i) * 32 + lane) * 16) : 0u;
    const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
    const int jrow = (hi16 ? 2 : 0) + (hi8 ? 1 : 0);  // the row of four whose sum fold4 leaves on this lane
    auto block_of = [&](int row) { return (int)(((A.row0 + row_a + row) >> p.bn_shift) - srow_lo); };
    float f[GT][C];
    int blk = -1;  // scale row the factors f are for
    RingPos rp;
    for (int it = 0; it < items; ++it, rp.next(NS)) {
        const int s = rp.s, r0 = it * R, nr = min(R, rows - r0);
        const bool landed = mbar_wait(full0 + s * 8, rp.ph, X.status);  // false: a wait gave up, the step is void
        const uint32_t sbase = stage0 + s * p.stage_bytes;
        for (int r = grp; r < nr && landed && grp < G; r += 4 * G) {  // four rows at a time: r, r + G, r + 2G, r + 3G
            uint32_t ra[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) ra[j] = sbase + min(r + j * G, nr - 1) * p.k;
            const int mine = r + jrow * G, b_last = block_of(r0 + min(r + 3 * G, nr - 1));
            // once, or once more for each further scale row that the four rows reach into
            for (int b = block_of(r0 + r); b <= b_last; ++b) {
                if (b != blk) {
                    blk = b;
#pragma unroll
                    for (int i = 0; i < C; ++i) {
                        const float sw = sw_s[b * p.skb + swc[i]];
#pragma unroll
                        for (int t = 0; t < GT; ++t) f[t][i] = live[i] ? sa[t][i] * sw : 0.0f;
                    }
                }
                float acc[GT][4];
#pragma unroll
                for (int i = 0; i < C; ++i) {
                    uint4 w[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[j] = lds_u128(ra[j] + off[i]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t ww[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
                        float s0[GT], s1[GT];
#pragma unroll
                        for (int t = 0; t < GT; ++t) s0[t] = s1[t] = 0.0f;
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const uint32_t h0 = e4m3x2_half_to_f16x2<0>(ww[q]), h1 = e4m3x2_half_to_f16x2<1>(ww[q]);
#pragma unroll
                            for (int t = 0; t < GT; ++t) {
                                fma2_f16(s0[t], h0, xh[t][i][2 * q]);
                                fma2_f16(s1[t], h1, xh[t][i][2 * q + 1]);
                            }
                        }
#pragma unroll
                        for (int t = 0; t < GT; ++t) acc[t][j] = i == 0 ? (s0[t] + s1[t]) * f[t][i] : fmaf(s0[t] + s1[t], f[t][i], acc[t][j]);
                    }
                }
#pragma unroll
                for (int t = 0; t < GT; ++t) {
                    const float v = fold4(acc[t], hi16, hi8);
                    if ((lane & 7) == 0 && mine < nr && block_of(r0 + mine) == b) part_s[(t * S + slice) * p.rows_max + r0 + mine] = v;
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + s * 8);
    }
    consumer_bar();  // part_s complete

    auto value = [&](int tok, int r) {
        const float *q = part_s + (size_t)tok * S * p.rows_max + r;
        float v = q[0];
        for (int s = 1; s < S; ++s) v += q[s * p.rows_max];
        return v;
    };
    fp8_finish<CT>(p, A, X, seq, tid, rows, [&](int i) { return row_a + i; }, value);
}

template <int GT, int C>
__global__ void __launch_bounds__(kThreads, GT * C <= 4 ? 2 : 1) fp8_gemv_kernel(const __grid_constant__ Fp8GemvParams p) {
    const RankCtx &X = p.r[blockIdx.y].ctx;
    fp8_gemv_body<GT, C>(p);
    if (p.world > 1 || p.mode == kModeLmHead) step_end(X, step_begin(X), gridDim.x);  // a lone all-reduce rank exchanges nothing
    host_done_signal(X, gridDim.x);
}

}  // namespace ws

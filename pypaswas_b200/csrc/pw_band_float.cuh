// pw_band_float.cuh -- the band direction sweep of traced pairs with fp32
// scores (a score or penalty that is no whole number, or values past 2^24).
//
// As pw_band.cuh: one warp a 256-row band, 8 rows a lane, one column a step, the
// bands of a pair chained across warps with a published progress count; cell
// codes in the band layout (warp_layout_offset) and the pair's candidates.
// Every add and compare is the strip sweep's (sweep_dirs<float>), in the
// reference's operation order, so codes and scores are the same bits.
//
// Why: the strip sweep runs one lane a pair, 32 pairs a warp.  A few hundred
// traced pairs then fill a few dozen warps, each at the latency of its longest
// pair, one strip class after another (1,609 reads of 71-251 against adapters:
// 3.6 ms; 0.17 ms here, a warp a pair).
#pragma once
#include "pw_band.cuh"

namespace pw {

__host__ __device__ __forceinline__ int band_float_warp_smem(int alpha1) { return alpha1 * 2 * kWarp * 16; }

template <bool AFFINE>
__global__ void __launch_bounds__(128, 4) band_float_kernel(KernelArgs A, BandArgs B) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int alpha1 = A.P.alpha + 1;
    float4* prof = (float4*)(smem + wib * band_float_warp_smem(alpha1));  // [residue][rows 0-3, 4-7][lane]
    const float gap = A.P.gap_f, ext = A.P.ext_f, ge = A.P.ge_f, neg = -1.0e10f;

    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(B.counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= B.n_entries) break;
        const int4 en = B.entries[it];
        const BandPair BP = B.pairs[en.x];
        const int band = en.y, pred = en.z;
        const int q = BP.q, t = BP.t;
        const int lq = A.q.len[q], lt = A.t.len[t];
        // threshold of the pair (default_main.cu:609, SmithWatermanCuda.py:269-275)
        const float maxf = A.pair_max[(int64_t)q * A.pm_lane + (int64_t)t * A.pm_strip];
        const float pos = (float)(A.P.highest * (double)(lq < lt ? lq : lt) * A.P.filter_factor);
        const float thr = fmaxf(__fmul_rn(A.P.lower_limit, maxf), pos);
        if (band == 0 && lane == 0) {
            PairMeta& pm = A.metas[BP.slot];
            pm.query = q;
            pm.target = t;
            pm.item = BP.meta_item;
            pm.lane = 0;
            pm.thr_f = thr;
            pm.thr_i = 0;
            pm.max_f = maxf;
        }
        Cand* cand = A.cands + A.cand_base[BP.slot];
        const int cap = A.cand_cap[BP.slot];
        int* ncand = A.n_cand + BP.slot;
        const uint8_t* qg = A.q.codes + A.q.code_off[q];
        const int64_t nsteps = (int64_t)lq + kWarp - 1;
        const int ymine = band * kBandRows + lane * kWarpRows;
        __syncwarp();
        {
            const uint8_t* tr = A.t.codes + A.t.code_off[t] + ymine;
            for (int a = 0; a < alpha1; ++a) {
                float w[kWarpRows];
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r) w[r] = ymine + r < lt ? A.cmat_f[a * A.P.dim + tr[r]] : -1.0e30f;
                prof[2 * a * kWarp + lane] = make_float4(w[0], w[1], w[2], w[3]);
                prof[(2 * a + 1) * kWarp + lane] = make_float4(w[4], w[5], w[6], w[7]);
            }
        }
        __syncwarp();
        const bool has_up = band > 0, has_down = band + 1 < BP.nbands;
        const float4* ring_in = (const float4*)B.ring + BP.ring_off + (int64_t)((band + 1) & 1) * lq;
        float4* ring_out = (float4*)B.ring + BP.ring_off + (int64_t)(band & 1) * lq;
        const int* prog_in = B.progress + pred;
        int* prog_out = B.progress + it;
        uint8_t* codes = A.codes + BP.dir_base;
        const int rows_left = lt - ymine;  // rows r < rows_left of this lane lie inside the target
        // linear: H; affine: M, J (gaps along the columns), best
        float Hl[kWarpRows], Jl[kWarpRows], Bl[kWarpRows];
#pragma unroll
        for (int r = 0; r < kWarpRows; ++r) {
            Hl[r] = 0.0f;
            Jl[r] = neg;
            Bl[r] = 0.0f;
        }
        float bt_h = 0.0f, bt_i = neg, bt_b = 0.0f;  // the bottom row's H (M), I and best
        float up_h = 0.0f, up_b = 0.0f;              // the row above at the previous column
        const float4 none = make_float4(0.0f, neg, 0.0f, 0.0f);
        float4 cur = none, nxt = none;  // the row above, 32 columns at a time, a block ahead
        auto fetch = [&](int64_t c) -> float4 { return c < lq ? __ldcg(ring_in + c) : none; };
        int avail = 0;
        bool ok = true;
        for (int64_t s = 0; s < nsteps; ++s) {
            if (has_up && (s & 31) == 0) {
                // this block and the next one must be stored by the band above
                const int need = (int)(s + 64 < (int64_t)lq ? s + 64 : (int64_t)lq);
                if (avail < need) {
                    avail = chain_wait(prog_in, need, B.abort_flag, B.wait_ns);
                    if (avail < 0) {
                        ok = false;
                        break;
                    }
                }
                cur = s == 0 ? fetch(s + lane) : nxt;
                nxt = fetch(s + 32 + lane);
            }
            const int x = (int)s - lane;
            const bool active = x >= 0 && x < lq;
            float rh = __shfl_up_sync(0xffffffffu, bt_h, 1);
            float ri = neg, rb = 0.0f;
            if constexpr (AFFINE) {
                ri = __shfl_up_sync(0xffffffffu, bt_i, 1);
                rb = __shfl_up_sync(0xffffffffu, bt_b, 1);
            }
            float4 above = none;
            if (has_up) {
                above.x = __shfl_sync(0xffffffffu, cur.x, (int)(s & 31));
                if constexpr (AFFINE) {
                    above.y = __shfl_sync(0xffffffffu, cur.y, (int)(s & 31));
                    above.z = __shfl_sync(0xffffffffu, cur.z, (int)(s & 31));
                }
            }
            if (lane == 0) {
                rh = active ? above.x : 0.0f;
                ri = active ? above.y : neg;
                rb = active ? above.z : 0.0f;
            }
            const float dg_h = x == 0 ? 0.0f : up_h, dg_b = x == 0 ? 0.0f : up_b;
            up_h = rh;
            up_b = rb;
            if (active) {
                const int a = __ldg(qg + x);
                const float4 p0 = prof[2 * a * kWarp + lane], p1 = prof[(2 * a + 1) * kWarp + lane];
                const float sc[kWarpRows] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
                // the stop flag needs a cell inside the matrix: x > 0 and y > 0
                const uint32_t stop = x > 0 ? kUL | kStopFlag : (uint32_t)kUL;
                const uint32_t stop0 = ymine > 0 ? stop : (uint32_t)kUL;
                uint32_t w = 0;
                float top = 0.0f;
                if constexpr (!AFFINE) {
                    float up = rh, diag = dg_h;
#pragma unroll
                    for (int r = 0; r < kWarpRows; ++r) {
                        const float left = Hl[r], ls = left + gap, us = up + gap;
                        const float h = fmaxf(fmaxf(us, fmaxf(ls, diag + sc[r])), 0.0f);
                        uint32_t cd = diag == 0.0f ? (r > 0 ? stop : stop0) : (uint32_t)kUL;
                        cd = h == us ? (uint32_t)kUp : cd;
                        cd = h == ls ? (uint32_t)kLeft : cd;
                        w |= (h > 0.0f ? cd : 0u) << (4 * r);
                        diag = left;
                        Hl[r] = h;
                        up = h;
                        top = fmaxf(top, h);
                    }
                    bt_h = up;
                } else {
                    float mup = rh, iup = ri, bdiag = dg_b, mdiag = dg_h;
#pragma unroll
                    for (int r = 0; r < kWarpRows; ++r) {
                        const float m = fmaxf(bdiag + sc[r], 0.0f);
                        const float i = fmaxf(iup + ext, mup + ge);
                        const float j = fmaxf(Jl[r] + ext, Hl[r] + ge);
                        const float b = fmaxf(fmaxf(m, i), j);
                        uint32_t cd = mdiag == 0.0f ? (r > 0 ? stop : stop0) : (uint32_t)kUL;
                        cd = b == m ? cd : b == i ? (uint32_t)kUp : (uint32_t)kLeft;
                        w |= (b > 0.0f ? cd : 0u) << (4 * r);
                        bdiag = Bl[r];
                        mdiag = Hl[r];
                        Hl[r] = m;
                        Jl[r] = j;
                        Bl[r] = b;
                        mup = m;
                        iup = i;
                        top = fmaxf(top, m);
                    }
                    bt_h = mup;
                    bt_i = iup;
                    bt_b = Bl[kWarpRows - 1];
                }
                if (top >= thr) {
                    // candidates: UL (MAIN) cells inside the matrix at or above the threshold
#pragma unroll
                    for (int r = 0; r < kWarpRows; ++r) {
                        if (Hl[r] < thr || r >= rows_left || ((w >> (4 * r)) & 3u) != kUL) continue;
                        w |= (uint32_t)kCand << (4 * r);
                        const int k = atomicAdd(ncand, 1);
                        if (k < cap) {
                            Cand cc;
                            cc.x = x;
                            cc.y = ymine + r;
                            cc.score_i = (int32_t)Hl[r];
                            cc.score_f = Hl[r];
                            cand[k] = cc;
                        }
                    }
                }
                *(uint32_t*)(codes + ((band * nsteps + s) * kWarp + lane) * kWarpRows / 2) = w;
                if (lane == kWarp - 1 && has_down) __stcg(ring_out + x, make_float4(bt_h, bt_i, bt_b, 0.0f));
            } else {
                // not started (x < 0): hand the left-boundary values down
                bt_h = 0.0f;
                bt_i = neg;
                bt_b = 0.0f;
            }
            // lane 31 stored columns 0 .. s - 31 of the bottom row
            if (has_down && lane == kWarp - 1 && ((s + 1) & 31) == 0 && s >= kWarp - 1)
                st_release_gpu(prog_out, (int)(s - (kWarp - 2)));
        }
        if (!ok) break;
        if (has_down && lane == kWarp - 1) st_release_gpu(prog_out, lq);
        // the band above has finished: its candidates are final
        if (has_up && chain_wait(prog_in, kChainDone, B.abort_flag, B.wait_ns) < 0) break;
        if (has_down)
            chain_publish(prog_out, kChainDone);
        else if (lane == 0)
            A.metas[BP.slot].n_cand = atomicAdd(ncand, 0);
    }
}

}  // namespace pw

// pw_band_affine.cuh -- the band sweep of single pairs, affine gap: pair maxima
// (DIRS 0: listed pairs, few long sequences, the unbatched form) or cell codes
// and candidates of traced pairs (DIRS 1), exactly as the strip sweeps compute
// them.
//
// One warp sweeps a 256-row band, the bands of a pair chained across warps as
// in pw_band.cuh.  A lane owns 8 rows and sweeps blocks of 2 columns, lane l one
// block behind lane l - 1: what a step costs besides its cells is shared by
// both columns, while the 62 columns that the lanes' skew adds to a band stay
// small against a protein (with 4 columns a block they would be 124).
//
// What bounds it: the ALU pipe.  M + s, M + gap + ext and the addresses are
// plain adds, the gap chains one DPX add-max each, B one three-way maximum with
// its floor at 0 (M itself is not floored: what a gap opened from a negative M
// differs in is negative, and B >= 0 never sees it; M's sign decides the stop
// flag).  Codes take four compares and selects a cell.  Candidates are looked
// for only in a column whose maximum reaches the threshold.
//
// Handing a row down: lane 31 stores its bottom row block by block into the
// pair's ring (band b: row b % rows), each word with the band's epoch in its top
// 6 bits; the ring is zeroed before the launch.  A word that shows the epoch is
// the band's, so neither side fences: the band below loads 16 blocks ahead and
// polls, bounded in time, while a word is missing.  All bands of a pair may be
// in flight together, so a band may poll a row whose band has not been taken
// yet: rows, epochs and the wait of a band for an earlier one to finish (the
// queue entry's w) are such that no word of another band ever shows the epoch
// waited for (affine_hold, pw_plan.h).
//   word 0 of a column: B (< 2^24) | (M <= 0) << 25 | epoch << 26
//   word 1: Y of the row below + 2^24 | epoch << 26
//
// Cell codes: [band][step][lane][2 columns][8 rows] nibbles (affine_layout_offset,
// pw_kernels.cuh), 8 bytes a lane and step, 256 contiguous bytes a warp.
//
// Before a lane's first block everything it computes from padding codes is
// negative or 0, after its last one values only decay, so no step is predicated
// except the stores.
#pragma once
#include "pw_band.cuh"
#include "pw_band_ck.cuh"
#include "pw_plan.h"

namespace pw {

constexpr int kAffCols = 2;    // columns a lane sweeps per step
constexpr int kAffGroup = 16;  // steps between two loads of the row above
constexpr int kAffLead = 56;   // planning lead between bands (steps)
constexpr int kAffMz = 1 << 25;

__host__ __device__ __forceinline__ int affine_blocks(int lq) { return (lq + kAffCols - 1) / kAffCols; }
__host__ __device__ __forceinline__ int band_affine_warp_smem(int alpha1) {
    // profile, the row above's blocks, code pairs of the last 64 blocks
    return alpha1 * kWarp * 8 + kAffGroup * 16 + 2 * kWarp * 2;
}
// Warps in flight an SM for `bands` bands of `pairs` pairs on `sms` SMs: a block
// of 4 for each four bands a warp, up to the 4 that fit, and two at least for
// short chains (fewer than 3 bands a pair).  A chain goes at the pace of its most
// crowded band, so that more blocks than the bands need make all of them wait;
// one warp alone keeps a sub-partition's ALU pipe 40% busy, four 85%.  Cell
// codes, with 4 blocks and with 1 / 2, proteins of 2 to 8 thousand residues: 48
// pairs (900 bands) 3.3 and 2.2 / 3.3 ms, 96 5.9 and 3.4 / 3.6, 200 (3600) 7.2
// and 7.3 / 5.8, 300 9.3 and 10.4 / 8.9, 500 14.1 and 16.9 / 13.8; two bands a
// pair: 1200 pairs .38 and .43 / .32; the 12,600 traced pairs of a 200 x 2000
// protein batch 5.2 and 9.2 / 6.5.
inline int band_affine_sm_warps(int64_t bands, int64_t pairs, int sms) {
    const int64_t blocks = 1 + bands / (16 * sms);
    return 4 * (int)std::min<int64_t>(bands < 3 * pairs ? std::max<int64_t>(blocks, 2) : blocks, 4);
}

template <int DIRS>
__global__ void __launch_bounds__(128, 4) band_affine_kernel(KernelArgs A, BandArgs B) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int alpha1 = A.P.alpha + 1;
    unsigned char* base = smem + wib * band_affine_warp_smem(alpha1);
    uint2* prof = (uint2*)base;                              // [residue][lane] -> 8 int8 scores
    uint4* above = (uint4*)(base + alpha1 * kWarp * 8);      // the row above's blocks of this group
    uint16_t* codes = (uint16_t*)(above + kAffGroup);        // code pairs of the last 64 blocks
    const int ext = A.P.ext_i, ge = A.P.ge_i;
    const uint32_t pad2 = (uint32_t)(alpha1 - 1) * 0x0101u;

    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(B.counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= B.n_entries) break;
        const int4 en = B.entries[it];
        const BandPair BP = B.pairs[en.x];
        const int band = en.y, pred = en.z, held = en.w;
        const int q = BP.q, t = BP.t;
        const int lq = A.q.len[q], lt = A.t.len[t];
        const int nblk = affine_blocks(lq);
        const bool has_up = band > 0, has_down = band + 1 < BP.nbands;
        int thr = 0, cap = 0;
        Cand* cand = nullptr;
        int* ncand = nullptr;
        if constexpr (DIRS == 1) {
            // threshold of the pair (default_main.cu:609, SmithWatermanCuda.py:269-275)
            const float maxf = A.pair_max[(int64_t)q * A.pm_lane + (int64_t)t * A.pm_strip];
            const int mn = lq < lt ? lq : lt;
            const float pos = (float)(A.P.highest * (double)mn * A.P.filter_factor);
            const float thf = fmaxf(__fmul_rn(A.P.lower_limit, maxf), pos);
            thr = (int)fminf(fmaxf(ceilf(thf), -1.0e9f), 1.0e9f);
            if (band == 0 && lane == 0) {
                PairMeta& pm = A.metas[BP.slot];
                pm.query = q;
                pm.target = t;
                pm.item = BP.meta_item;
                pm.lane = 0;
                pm.thr_f = thf;
                pm.thr_i = thr;
                pm.max_f = maxf;
            }
            cand = A.cands + A.cand_base[BP.slot];
            cap = A.cand_cap[BP.slot];
            ncand = A.n_cand + BP.slot;
        }
        const uint16_t* qw = (const uint16_t*)(A.q.codes + A.q.code_off[q]);
        const int ymine = band * kBandRows + lane * kWarpRows;
        __syncwarp();
        {
            uint8_t res[kWarpRows];
            const uint8_t* tr = A.t.codes + A.t.code_off[t] + ymine;
#pragma unroll
            for (int r = 0; r < kWarpRows; ++r) res[r] = ymine + r < lt ? tr[r] : 0;
            for (int a = 0; a < alpha1; ++a) {
                uint32_t w[2] = {0u, 0u};
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r) {
                    const int8_t sc = ymine + r < lt ? A.cmat_i8[a * A.P.dim + res[r]] : (int8_t)-128;
                    w[r / 4] |= (uint32_t)(uint8_t)sc << (8 * (r % 4));
                }
                prof[a * kWarp + lane] = make_uint2(w[0], w[1]);
            }
        }
        // code pairs are staged a group ahead of their use
        auto load_code = [&](int first) -> uint32_t {
            return lane < kAffGroup && first + lane < nblk ? qw[first + lane] : pad2;
        };
        codes[lane] = (uint16_t)pad2;
        codes[lane + kWarp] = (uint16_t)pad2;
        __syncwarp();
        if (lane < kAffGroup) codes[lane] = (uint16_t)load_code(0);
        uint32_t code_n = load_code(kAffGroup);
        // (the row of band 0 - 1 is not read)
        const int rows = BP.rows;
        const uint4* in = (const uint4*)B.ring + BP.ring_off + (int64_t)((band + rows - 1) % rows) * nblk;
        uint4* out = (uint4*)B.ring + BP.ring_off + (int64_t)(band % rows) * nblk;
        const uint32_t ep_in = (has_up ? affine_epoch(band - 1, rows) : 0u) << 26;
        const uint32_t ep_out = affine_epoch(band, rows) << 26;
        // an earlier band whose words must be gone from the row above
        if (held >= 0 && chain_wait(B.progress + held, kChainDone, B.abort_flag, B.wait_ns) < 0) break;
        // the row above band 0 (and past the query): B = 0, Y = -inf
        const uint4 none = make_uint4(ep_in, ep_in, ep_in, ep_in);
        auto load_above = [&](int first) -> uint4 {
            if (has_up && lane < kAffGroup && first + lane < nblk) return ld_relaxed_v4(in + first + lane);
            return none;
        };
        auto stored = [&](uint4 v) -> bool {  // every word shows the band's epoch
            return (((v.x ^ ep_in) | (v.y ^ ep_in) | (v.z ^ ep_in) | (v.w ^ ep_in)) >> 26) == 0u;
        };
        uint4 above_n = load_above(0);
        int Bl[kWarpRows], Zl[kWarpRows], Ml[kWarpRows];
#pragma unroll
        for (int r = 0; r < kWarpRows; ++r) {
            Bl[r] = 0;
            Zl[r] = kNeg;
            Ml[r] = 0;
        }
        // the row above over this step's block, from the lane above a step ago
        int up_b[kAffCols] = {0, 0}, up_y[kAffCols] = {kNeg, kNeg};
        int b_prev = 0;  // word 0 of the row above at the column before this block
        int mx = 0;
        uint8_t* cell_codes = DIRS == 1 ? A.codes + BP.dir_base : nullptr;
        const int nsteps = nblk + kWarp - 1;
        __syncwarp();
        uint32_t word = codes[(-lane) & 63];
        bool ok = true;
        for (int first = 0; first < nsteps; first += kAffGroup) {
            if (has_up) {
                // this group's blocks of the row above must be stored
                unsigned long long began = 0;
                unsigned ns = 32;
                while (!__all_sync(0xffffffffu, stored(above_n))) {
                    const unsigned long long now = global_ns();
                    if (began == 0) began = now;
                    const bool give_up = ld_acquire_gpu(B.abort_flag) != 0 || now - began > B.wait_ns;
                    if (__any_sync(0xffffffffu, give_up)) {
                        if (lane == 0) atomicExch(B.abort_flag, 1);
                        ok = false;
                        break;
                    }
                    __nanosleep(ns);
                    if (ns < 256) ns <<= 1;
                    above_n = load_above(first);
                }
                if (!ok) break;
            }
            __syncwarp();  // the last group's reads are done
            if (lane < kAffGroup) {
                const uint32_t m = (1u << 26) - 1u;
                // Y: - 2^24, and -inf where nothing was stored (0 stands for it)
                const int y0 = (int)(above_n.y & m) - (1 << 24), y1 = (int)(above_n.w & m) - (1 << 24);
                above[lane] = make_uint4(above_n.x & m, (uint32_t)y0, above_n.z & m, (uint32_t)y1);
                codes[(first + kAffGroup + lane) & 63] = (uint16_t)code_n;
            }
            __syncwarp();
            code_n = load_code(first + 2 * kAffGroup);
            above_n = load_above(first + kAffGroup);
            const int last = min(first + kAffGroup, nsteps);
#pragma unroll 1
            for (int st = first; st < last; ++st) {
                const int k = st - lane;  // this lane's block
                if (lane == 0) {
                    const uint4 v = above[st & (kAffGroup - 1)];
                    up_b[0] = (int)v.x;
                    up_y[0] = (int)v.y;
                    up_b[1] = (int)v.z;
                    up_y[1] = (int)v.w;
                }
                uint2 pw[kAffCols];
#pragma unroll
                for (int j = 0; j < kAffCols; ++j) pw[j] = prof[((word >> (8 * j)) & 0xff) * kWarp + lane];
                word = codes[(k + 1) & 63];
                uint32_t w[kAffCols] = {0u, 0u};
                int dn_b[kAffCols], dn_y[kAffCols];
#pragma unroll
                for (int j = 0; j < kAffCols; ++j) {
                    const int above_w = j == 0 ? b_prev : up_b[j - 1];
                    int bd = above_w & (kAffMz - 1);        // B one row up, one column back
                    int md = above_w & kAffMz ? 0 : 1;      // M there (its sign)
                    int y = up_y[j];
                    // the stop flag needs a cell inside the matrix
                    const uint32_t stop = 2 * k + j > 0 ? kUL | kStopFlag : (uint32_t)kUL;
                    const uint32_t stop0 = ymine > 0 ? stop : (uint32_t)kUL;
#pragma unroll
                    for (int r = 0; r < kWarpRows; ++r) {
                        const int m = bd + prof_score(pw[j], r);
                        const int xg = Zl[r];
                        const int b = __vimax3_s32_relu(m, y, xg);
                        if constexpr (DIRS == 1) {
                            // the reference's classification: MAIN when B == M, else I (Y), else J (X)
                            uint32_t cd = md <= 0 ? (r > 0 ? stop : stop0) : (uint32_t)kUL;
                            const uint32_t gp = b == y ? (uint32_t)kUp : (uint32_t)kLeft;
                            cd = b == m ? cd : gp;
                            cd = b > 0 ? cd : 0u;
                            w[j] += cd << (4 * r);
                            md = Ml[r];
                            Ml[r] = m;
                        }
                        const int mg = m + ge;
                        Zl[r] = addmax(xg, ext, mg);
                        y = addmax(y, ext, mg);
                        bd = Bl[r];
                        Bl[r] = b;
                    }
                    const int smax = max3(max3(Bl[0], Bl[1], Bl[2]), max3(Bl[3], Bl[4], Bl[5]), max(Bl[6], Bl[7]));
                    if constexpr (DIRS == 0) {
                        mx = max(mx, smax);
                    } else if (smax >= thr) {
                        const int x = 2 * k + j;
#pragma unroll
                        for (int r = 0; r < kWarpRows; ++r) {
                            if (Bl[r] < thr || ((w[j] >> (4 * r)) & 3u) != kUL || x >= lq || k < 0 || ymine + r >= lt)
                                continue;
                            w[j] |= (uint32_t)kCand << (4 * r);
                            const int c = atomicAdd(ncand, 1);
                            if (c < cap) {
                                Cand cc;
                                cc.x = x;
                                cc.y = ymine + r;
                                cc.score_i = Bl[r];
                                cc.score_f = (float)Bl[r];
                                cand[c] = cc;
                            }
                        }
                    }
                    dn_b[j] = Bl[kWarpRows - 1] | (DIRS == 1 && Ml[kWarpRows - 1] <= 0 ? kAffMz : 0);
                    dn_y[j] = y;
                }
                b_prev = up_b[kAffCols - 1];
                if (has_down && lane == kWarp - 1 && k >= 0)
                    st_relaxed_v4(out + k, make_uint4((uint32_t)dn_b[0] | ep_out, (uint32_t)(dn_y[0] + (1 << 24)) | ep_out,
                                                      (uint32_t)dn_b[1] | ep_out, (uint32_t)(dn_y[1] + (1 << 24)) | ep_out));
                if (DIRS == 1 && (unsigned)k < (unsigned)nblk)
                    *(uint2*)(cell_codes + (((int64_t)band * nsteps + st) * kWarp + lane) * 8) = make_uint2(w[0], w[1]);
#pragma unroll
                for (int j = 0; j < kAffCols; ++j) {
                    up_b[j] = __shfl_up_sync(0xffffffffu, dn_b[j], 1);
                    up_y[j] = __shfl_up_sync(0xffffffffu, dn_y[j], 1);
                }
            }
        }
        if (!ok) break;
        if constexpr (DIRS == 0) mx = __reduce_max_sync(0xffffffffu, mx);
        if (has_up) {
            // the band above has finished: its running maximum and its candidates are final
            if (chain_wait(B.progress + pred, kChainDone, B.abort_flag, B.wait_ns) < 0) break;
            if constexpr (DIRS == 0) mx = max(mx, __ldcg(&B.run_max[pred]));
        }
        if (has_down) {
            if constexpr (DIRS == 0)
                if (lane == 0) __stcg(&B.run_max[it], mx);
            chain_publish(B.progress + it, kChainDone);
        } else if (lane == 0) {
            if constexpr (DIRS == 1)
                A.metas[BP.slot].n_cand = atomicAdd(ncand, 0);
            else
                B.max_out[BP.slot] = (float)mx;
        }
    }
}

}  // namespace pw

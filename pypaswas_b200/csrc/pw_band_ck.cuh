// pw_band_ck.cuh -- the score sweep of listed long pairs (linear gap), which
// also keeps the tile form's checkpoints and tile maxima (pw_tiles.cuh).
//
// One warp sweeps a 256-row band, the bands of a pair chained across warps as
// in pw_band.cuh.  PAIR: two listed pairs that share their query and whose
// targets have the same length (a pair and the pair with the target's reverse
// complement) run as one sweep with each cell's two H values in the low and
// high 16-bit halves of one register; otherwise one pair on 32-bit lanes.
//
// What bounds it, and why this shape.  A lane owns 8 rows and sweeps blocks of
// 4 columns, lane l one block behind lane l - 1, so that what a step costs
// besides its cells -- the boundary values from the lane above (4 shuffles),
// the code word, the loop -- is paid once for 32 cells (one column a step took
// 154 instructions for 8 cells, ~900 clocks a step with one warp on an SM).
// The cells themselves: per row 2 DPX on the ALU pipe, a packed add on the FMA
// pipe, half a three-way maximum.  The profile is [residue][half][lane] in
// 16-byte entries: a lane reads its own 8 rows' scores without bank conflicts
// whatever its residue.
//
// Handing a row down: the bottom row of a band is stored block by block (16
// bytes: 4 columns) into its checkpoint row with bit 31 of every word set, and
// the rows are zeroed before the sweep.  A word that shows the bit is valid by
// itself, so neither side fences: the band below loads 8 blocks ahead (lanes 0
// to 7, one coalesced access) and polls only while a word is still missing
// (the release and acquire of a progress count, every 16 columns, stalled the
// storing warp for the latency of its outstanding stores each time).  Each
// poll is bounded in time, as every wait here.
//
// Blocks per SM (kBandCkBlocks, band_ck_sm_warps).  A chain goes at the pace of
// its slowest band, the one whose SM sub-partition has most warps at work, and
// one warp alone keeps the ALU pipe three quarters busy: with 4 blocks of 4
// warps an SM, bands waited for the band above 40% of their time and the pipe
// was 66% busy.  64 pairs of 10 to 50 kb (3900 bands): 17.6 ms with 4 blocks,
// 15.9 with 3, 15.1 with 2, 17.4 with 1.  With few bands one block an SM is
// better, all bands then going at one pace; pairs of 20 to 30 kb with 1 and 2
// blocks: 8 pairs 2.7 and 4.2 ms, 16 3.7 and 4.6, 24 (2350 bands) 5.1 and 5.3,
// 32 (3100) 6.9 and 6.7; the line is drawn at four bands a warp.  Blocks of 8
// columns a lane (half the steps, twice the skew) were slower: 16.1 ms for the
// 64 pairs.
//
// Steps past a lane's ends run on padding codes: before its first block H
// stays 0, after its last one it only decays, so no step is predicated except
// the stores.
//
// A block's columns past the query hold decayed values; checkpoint rows are
// (lq + 3) & ~3 wide and nothing reads those columns.
//
// 16-bit halves hold H exactly while every value stays at or below 32767 - the
// matrix's highest score (no add can then wrap); a pair whose maximum passes that
// limit is reported in `over` and swept again on 32-bit lanes by the host.
#pragma once
#include "pw_band.cuh"

namespace pw {

struct BandCk {
    int32_t q;            // the query
    int32_t t[2];         // targets of the low and high halves (same length); single: t[0]
    int32_t nbands;
    int64_t slot[2];      // pair-list indices (maxima)
    int64_t rows;         // int offset of the checkpoint rows ((nbands - 1) x tile_row_stride)
    int64_t cols;         // int offset of the checkpoint columns (nbands x tiles x 256)
    int64_t tm[2];        // int offsets of the pairs' tile maxima (nbands x tiles)
};

struct BandCkArgs {
    const int4* entries;  // per queue entry: (pair, band, queue index of the band above, 0)
    const BandCk* pairs;
    int n_entries;
    int* counter;
    int* progress;        // per entry: kChainDone when finished
    int2* run_max;        // per entry: running maxima of the two pairs' bands so far
    int* abort_flag;
    float* max_out;       // pair maxima, indexed by BandCk.slot
    int* over;            // PAIR: per pair-list index, 1 when its maximum passed the 16-bit limit
    int* ck;              // checkpoints and tile maxima
    int limit;            // PAIR: 32767 - the matrix's largest absolute score
    unsigned long long wait_ns;
};

constexpr int kBlkCols = 4;   // columns a lane sweeps per step
constexpr int kBlkGroup = 8;  // steps between two loads of the row above
constexpr int kBandCkBlocks = 2; // blocks of 4 warps an SM at most
constexpr int kBandCkLead = 48;  // planning lead between bands (steps): the lanes' skew, a group and the hand-over

__host__ __device__ __forceinline__ int band_ck_warp_smem(int alpha1) {
    // profile, the row above's blocks, the tile's last column, its maxima, code words
    return alpha1 * 2 * kWarp * 16 + kBlkGroup * 16 + 2 * kWarp * 16 + kWarp * 4 + 2 * kWarp * 4;
}

// Warps in flight an SM for `bands` bands on `sms` SMs.
inline int band_ck_sm_warps(int64_t bands, int sms) { return bands < (int64_t)4 * 4 * sms ? 4 : 4 * kBandCkBlocks; }

__device__ __forceinline__ int lo16(uint32_t v) { return (int)(int16_t)(v & 0xffffu); }
__device__ __forceinline__ int hi16(uint32_t v) { return (int)(int16_t)(v >> 16); }

__device__ __forceinline__ uint4 ld_relaxed_v4(const uint4* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_v4(uint4* p, uint4 v) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};"
                 ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

constexpr uint32_t kRowTag = 0x80000000u;  // H is never negative: the bit marks a stored word

template <bool PAIR>
__device__ __forceinline__ uint32_t ck_max3(uint32_t a, uint32_t b, uint32_t c) {
    if constexpr (PAIR) return __vimax3_s16x2(a, b, c);
    return (uint32_t)__vimax3_s32((int)a, (int)b, (int)c);
}

// max(up + gap, left + gap, diag + s, 0)
template <bool PAIR>
__device__ __forceinline__ uint32_t ck_cell(uint32_t diag, uint32_t s, uint32_t left, uint32_t up, uint32_t gap) {
    if constexpr (PAIR)
        return __viaddmax_s16x2_relu(up, gap, __viaddmax_s16x2(left, gap, __vadd2(diag, s)));
    return (uint32_t)__viaddmax_s32_relu((int)up, (int)gap, __viaddmax_s32((int)left, (int)gap, (int)(diag + s)));
}

template <bool PAIR>
__global__ void __launch_bounds__(128, kBandCkBlocks) band_ck_kernel(KernelArgs A, BandCkArgs B) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int alpha1 = A.P.alpha + 1;
    unsigned char* base = smem + wib * band_ck_warp_smem(alpha1);
    uint4* prof = (uint4*)base;                      // [residue][rows 0-3, 4-7][lane]
    uint4* above = prof + alpha1 * 2 * kWarp;        // the row above's blocks of this group
    uint4* save = above + kBlkGroup;                 // a tile's last column, [rows 0-3, 4-7][lane]
    uint32_t* save_tm = (uint32_t*)(save + 2 * kWarp);  // its maximum, per lane
    uint32_t* codes = save_tm + kWarp;               // code words of the last 64 blocks
    const uint32_t gap = PAIR ? pack16(A.P.gap_i) : (uint32_t)A.P.gap_i;
    const uint32_t pad4 = (uint32_t)(alpha1 - 1) * 0x01010101u;

    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(B.counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= B.n_entries) break;
        const int4 en = B.entries[it];
        const BandCk BP = B.pairs[en.x];
        const int band = en.y, pred = en.z;
        const int lq = A.q.len[BP.q], lt = A.t.len[BP.t[0]];
        const int nblk = (lq + kBlkCols - 1) / kBlkCols;
        const bool has_up = band > 0, has_down = band + 1 < BP.nbands;
        const uint32_t* qw = (const uint32_t*)(A.q.codes + A.q.code_off[BP.q]);
        __syncwarp();
        {
            // this lane's 8 rows (rows past the target: -128)
            const int y0 = band * kBandRows + lane * kWarpRows;
            uint8_t r0[kWarpRows], r1[kWarpRows];
            const uint8_t* t0 = A.t.codes + A.t.code_off[BP.t[0]] + y0;
            const uint8_t* t1 = A.t.codes + A.t.code_off[BP.t[PAIR ? 1 : 0]] + y0;
#pragma unroll
            for (int r = 0; r < kWarpRows; ++r) {
                r0[r] = y0 + r < lt ? t0[r] : 0;
                r1[r] = PAIR && y0 + r < lt ? t1[r] : 0;
            }
            for (int a = 0; a < alpha1; ++a) {
                uint32_t w[kWarpRows];
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r) {
                    const int s0 = y0 + r < lt ? (int)A.cmat_i8[a * A.P.dim + r0[r]] : -128;
                    if constexpr (PAIR) {
                        const int s1 = y0 + r < lt ? (int)A.cmat_i8[a * A.P.dim + r1[r]] : -128;
                        w[r] = pack16x2(s0, s1);
                    } else {
                        w[r] = (uint32_t)s0;
                    }
                }
                prof[(2 * a) * kWarp + lane] = make_uint4(w[0], w[1], w[2], w[3]);
                prof[(2 * a + 1) * kWarp + lane] = make_uint4(w[4], w[5], w[6], w[7]);
            }
        }
        codes[lane] = pad4;
        codes[lane + kWarp] = pad4;
        const int64_t stride = tile_row_stride(lq);
        const uint4* in = (const uint4*)(B.ck + BP.rows + (int64_t)(band - 1) * stride);
        uint4* out = (uint4*)(B.ck + BP.rows + (int64_t)band * stride);
        const int ntiles = tile_count(lq);
        uint4* cols = (uint4*)(B.ck + BP.cols + (int64_t)band * ntiles * kBandRows + lane * kWarpRows);
        int* tmax0 = B.ck + BP.tm[0] + (int64_t)band * ntiles;
        int* tmax1 = B.ck + BP.tm[PAIR ? 1 : 0] + (int64_t)band * ntiles;
        // one group's blocks: lanes 0 .. 7 hold block first + lane's code word and row above
        auto load_code = [&](int first) -> uint32_t {
            return lane < kBlkGroup && first + lane < nblk ? qw[first + lane] : pad4;
        };
        auto load_above = [&](int first) -> uint4 {
            if (has_up && lane < kBlkGroup && first + lane < nblk) return ld_relaxed_v4(in + first + lane);
            return make_uint4(kRowTag, kRowTag, kRowTag, kRowTag);
        };
        uint32_t H[kWarpRows];
        uint32_t up[kBlkCols];  // the row above over this step's block, from the lane above a step ago
#pragma unroll
        for (int r = 0; r < kWarpRows; ++r) H[r] = 0u;
#pragma unroll
        for (int j = 0; j < kBlkCols; ++j) up[j] = 0u;
        uint32_t diag0 = 0u;  // the row above at the column before this block
        uint32_t tm = 0u;     // the lane's maximum in its current tile
        int m0 = 0, m1 = 0;   // the pairs' maxima over the finished tiles
        // the tile's maximum over the lanes, into the tile maxima
        auto tile_max = [&](int j, uint32_t v) {
            const int a = __reduce_max_sync(0xffffffffu, PAIR ? lo16(v) : (int)v);
            m0 = max(m0, a);
            if (lane == 0) tmax0[j] = a;
            if constexpr (PAIR) {
                const int b = __reduce_max_sync(0xffffffffu, hi16(v));
                m1 = max(m1, b);
                if (lane == 0) tmax1[j] = b;
            }
        };
        const int nsteps = nblk + kWarp - 1;
        // code words are staged a group ahead of their use
        if (lane < kBlkGroup) codes[lane] = load_code(0);
        uint32_t code_n = load_code(kBlkGroup);
        uint4 above_n = load_above(0);
        __syncwarp();
        uint32_t word = codes[(-lane) & 63];
        bool ok = true;
        for (int first = 0; first < nsteps && ok; first += kBlkGroup) {
            // this group's blocks of the row above must be stored
            if (has_up) {
                unsigned long long began = 0;
                unsigned ns = 32;
                while (!__all_sync(0xffffffffu, (above_n.x & above_n.y & above_n.z & above_n.w & kRowTag) != 0u)) {
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
            if (lane < kBlkGroup) {
                above[lane] = make_uint4(above_n.x & ~kRowTag, above_n.y & ~kRowTag, above_n.z & ~kRowTag,
                                         above_n.w & ~kRowTag);
                codes[(first + kBlkGroup + lane) & 63] = code_n;
            }
            __syncwarp();
            code_n = load_code(first + 2 * kBlkGroup);
            above_n = load_above(first + kBlkGroup);
            const int last = min(first + kBlkGroup, nsteps);
#pragma unroll 1
            for (int t = first; t < last; ++t) {
                const int k = t - lane;  // this lane's block
                if (lane == 0) {
                    const uint4 v = above[t & (kBlkGroup - 1)];
                    up[0] = v.x;
                    up[1] = v.y;
                    up[2] = v.z;
                    up[3] = v.w;
                }
                uint32_t sc[kBlkCols][kWarpRows];
#pragma unroll
                for (int j = 0; j < kBlkCols; ++j) {
                    const uint4* p = prof + ((word >> (8 * j)) & 0xff) * (2 * kWarp) + lane;
                    const uint4 p0 = p[0], p1 = p[kWarp];
                    sc[j][0] = p0.x, sc[j][1] = p0.y, sc[j][2] = p0.z, sc[j][3] = p0.w;
                    sc[j][4] = p1.x, sc[j][5] = p1.y, sc[j][6] = p1.z, sc[j][7] = p1.w;
                }
                word = codes[(k + 1) & 63];
                // the block's cells by anti-diagonals: the four columns' chains
                // of dependent instructions run side by side
                uint32_t d[kBlkCols] = {diag0, up[0], up[1], up[2]}, u[kBlkCols] = {up[0], up[1], up[2], up[3]};
                diag0 = up[3];
#pragma unroll
                for (int w = 0; w < kWarpRows + kBlkCols - 1; ++w)
#pragma unroll
                    for (int j = 0; j < kBlkCols; ++j) {
                        const int r = w - j;
                        if (r < 0 || r >= kWarpRows) continue;
                        const uint32_t left = H[r];
                        const uint32_t h = ck_cell<PAIR>(d[j], sc[j][r], left, u[j], gap);
                        if (r & 1) tm = ck_max3<PAIR>(tm, u[j], h);
                        d[j] = left;
                        u[j] = h;
                        H[r] = h;
                    }
#pragma unroll
                for (int j = 0; j < kBlkCols; ++j) up[j] = __shfl_up_sync(0xffffffffu, u[j], 1);
                if (has_down && lane == kWarp - 1 && k >= 0)
                    st_relaxed_v4(out + k, make_uint4(u[0] | kRowTag, u[1] | kRowTag, u[2] | kRowTag, u[3] | kRowTag));
                if ((k & 31) == 31 && (unsigned)k < (unsigned)nblk) {
                    // the last column of a tile, kept until every lane has reached it
                    save[lane] = make_uint4(H[0], H[1], H[2], H[3]);
                    save[kWarp + lane] = make_uint4(H[4], H[5], H[6], H[7]);
                    save_tm[lane] = tm;
                    tm = 0u;
                }
                if ((t & 31) == 30 && t >= 62) {
                    // tile j's last column is complete: the next tile's left boundary
                    const int j = (t - 62) >> 5;
                    if (j * 32 + 31 < nblk) {
                        if ((j + 1) * kTileW < lq) {
                            uint4* d = cols + (int64_t)(j + 1) * (kBandRows / 4);
                            __stcg(d, save[lane]);
                            __stcg(d + 1, save[kWarp + lane]);
                        }
                        tile_max(j, save_tm[lane]);
                    }
                }
            }
        }
        if (!ok) break;
        if (nblk & 31) tile_max(nblk >> 5, tm);  // the last tile, narrower
        if (has_up) {
            // the band above has finished: its running maxima are final
            if (chain_wait(B.progress + pred, kChainDone, B.abort_flag, B.wait_ns) < 0) break;
            const int2 pm = __ldcg(&B.run_max[pred]);
            m0 = max(m0, pm.x);
            m1 = max(m1, pm.y);
        }
        if (has_down) {
            if (lane == 0) __stcg(&B.run_max[it], make_int2(m0, m1));
            chain_publish(B.progress + it, kChainDone);
        } else if (lane == 0) {
            B.max_out[BP.slot[0]] = (float)m0;
            if constexpr (PAIR) {
                B.max_out[BP.slot[1]] = (float)m1;
                B.over[BP.slot[0]] = m0 > B.limit ? 1 : 0;
                B.over[BP.slot[1]] = m1 > B.limit ? 1 : 0;
            }
        }
    }
}

}  // namespace pw

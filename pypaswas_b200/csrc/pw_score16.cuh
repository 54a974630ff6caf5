// pw_score16.cuh -- the 16-bit score sweep: two pairs per lane.
//
// Pair maxima only (the engine's first phase).  Every 32-bit register holds
// the same DP cell of two different pairs as signed 16-bit halves, and the
// recurrences run on the DPX 16x2 instructions (__viaddmax_s16x2 and friends),
// which update two cells per instruction at the rate of one 32-bit update.
// A warp aligns two "strip" sequences (low and high halves) against up to 32
// "lane" sequences, one per lane.  Both halves of a lane read the same lane
// residue, so the strip profile stores ready-made 16x2 score pairs.  Which
// input set provides the strips and which the lanes is chosen per run by the
// host (pair maxima are symmetric in the two sequences, so either orientation
// gives the same maxima).
//
// What bounds it: the DPX instructions, 64 lanes a clock and SM on the ALU
// pipe.  A packed add (__vadd2) issues beside them on the FMA pipe at the same
// rate (measured: 64 lanes alone, 120 when it alternates with a DPX add-max),
// so the adds that need no maximum of their own leave the ALU pipe:
//   linear  diagonal + score; 2 DPX + 1 add a row pair (3 DPX before);
//           registers only, 6 warps a scheduler: 6.2 clocks a row, 7.5 before
//   affine  diagonal + score and M + gap + ext, with the floor at 0 in the
//           three-way maximum of B instead of in M; 3 DPX + 2 adds (5 DPX
//           before); 9.0 clocks a row, 12.4 before
// (plus half a three-way maximum a row for the pair maximum in both).
//
// Overflow: with every score in [-127, 127], no 16-bit operation can exceed
// 32767 while all cell values stay below kOvf16 (32640 = 32767 - 127).  A pair
// whose maximum reaches kOvf16 is reported as NaN and recomputed by the 32-bit
// sweep.
#pragma once
#include "pw_kernels.cuh"

namespace pw {

constexpr int kOvf16 = 32767 - 127;
constexpr uint32_t kNeg16x2 = 0xC000C000u;  // -16384 in both halves (boundary of the gap chains)

__device__ __forceinline__ uint32_t pack16(int v) { return ((uint32_t)v & 0xffffu) * 0x00010001u; }
__device__ __forceinline__ uint32_t pack16x2(int lo, int hi) {
    return ((uint32_t)lo & 0xffffu) | ((uint32_t)hi << 16);
}

// The profile's layout: which load fetches the scores of a lane's residue.
//   kPair128  one uint4 holds 4 rows (16x2 words): for alphabets whose
//             residues' uint4 fall into different bank groups (8 codes)
//   kPair64   one uint2 holds 2 rows: with more residues a quarter warp's
//             128-bit loads meet in a bank group about twice (20 amino acids),
//             a half warp's 64-bit loads less often
//   kDual     the dual-lane form: one uint2 holds 4 rows of plain 16-bit scores
//   kPair32   one word holds a row: no two residues of up to 32 share a bank
enum Form16 { kPair128 = 0, kPair64 = 1, kDual = 2, kPair32 = 3 };

struct Score16Args {
    const WorkItem* items;   // target = strip A, index = strip B (or -1), first/lanes index the lane order
                             // (chained launch: the items that the queue entries name)
    int n_items;
    int* counter;
    const uint8_t* lane_codes;   // compact lane-alphabet codes, 16-aligned, pad-coded tail
    const int64_t* lane_off;
    const int32_t* lane_len;
    const int32_t* lane_order;   // sorted position -> lane sequence
    const uint8_t* strip_res;    // strip residues as matrix indices, 16-aligned
    const int64_t* strip_off;
    const int32_t* strip_len;
    const int8_t* cmat;          // [(alpha + 1) * dim] scores lane residue x strip residue
    int alpha1, dim;
    int gap, ext;
    float* pair_max;
    int64_t stride_strip, stride_lane;  // pair_max[strip * stride_strip + lane * stride_lane]
    uint4* bnd_pool;
    int64_t bnd_slot;            // uint4 elements per warp slot (two boundary rows, see ring_row)
    // multi-strip launch with chains (score16_chain_kernel): per queue entry
    // (chain, strip, queue index of the chain's previous strip, item); strip -1
    // marks a whole item swept by one warp with its boundary in bnd_pool
    const int4* chain;
    const int64_t* ring_off;     // per chain: its two boundary rows (ring_row uint4 each) in `ring`
    uint4* ring;
    int* progress;               // per queue entry: columns whose boundary row is written (kChainDone when finished)
    uint32_t* run_max;           // per queue entry x 32 lanes: running 16x2 maximum of the chain so far
    int pad_code;                // lane code of the padding residue
    int* abort_flag;             // set when a wait runs out of time; every waiting warp then gives up
    int n_chain_items;           // host-side bookkeeping: entries of the chained launch
    int item_base;               // chained launch: first queue entry of this launch (entries [item_base, n_items))
    int* ovf_count;              // pairs reported as NaN (16-bit limit reached)
    unsigned long long wait_ns;  // bound of one chain wait
    // grid form of a one-strip class launch (no item list): item `it` is lane
    // group it / grid_n_strips (grid_lane_step lanes from the sorted position
    // it / grid_n_strips * grid_lane_step) against strip pair
    // grid_strips[it % grid_n_strips] (x: strip A, y: strip B or -1)
    const int2* grid_strips;     // null: items come from `items`
    int grid_n_strips;
    int grid_lane_step;          // 32, or 64 for the dual-lane form
    int grid_n_lane;             // lane sequences in the sorted order
};

// Rows a profile entry holds, entry bytes, and entries a residue: a residue's
// entries lie together, so that a column's loads differ by constants, and one
// entry of padding makes their number odd, so that residues differ in bank
// group as their codes do.
template <int FORM>
__host__ __device__ constexpr int prof_rows() { return FORM == kPair32 ? 1 : FORM == kPair64 ? 2 : 4; }
template <int FORM>
__host__ __device__ constexpr int prof_entry_bytes() {
    return FORM == kPair128 ? (int)sizeof(uint4) : FORM == kPair32 ? (int)sizeof(uint32_t) : (int)sizeof(uint2);
}
template <int S, int FORM>
__host__ __device__ constexpr int prof_stride() { return (S / prof_rows<FORM>()) | 1; }

// Bytes of one warp's profile (a multiple of 16) and of a block's four.
template <int S, int FORM>
__host__ __device__ constexpr int warp_profile_bytes(int alpha1) {
    return (alpha1 * prof_stride<S, FORM>() * prof_entry_bytes<FORM>() + 15) & ~15;
}
template <int S, int FORM>
__host__ __device__ constexpr int block_profile_bytes(int alpha1) { return 4 * warp_profile_bytes<S, FORM>(alpha1); }

// Profile of strip rows [y0, y0 + S): the scores of lane residue a, strip A in
// the low halves and strip B in the high halves (dual-lane form: strip A's
// plain 16-bit scores).  Rows past a strip's end get -128.
template <int S, int FORM>
__device__ __forceinline__ void build_profile16(unsigned char* prof, const int8_t* cmat, const uint8_t* ra,
                                                const uint8_t* rb, int y0, int la, int lb, int alpha1, int dim,
                                                int lane) {
    constexpr int R = prof_rows<FORM>(), G = S / R, stride = prof_stride<S, FORM>();
    const int n = G * alpha1;
    for (int idx = lane; idx < n; idx += kWarp) {
        const int a = idx / G, g = idx % G;
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int y = y0 + R * g + k;
            const int sa = y < la ? (int)cmat[a * dim + ra[y]] : -128;
            if constexpr (FORM == kDual) {
                w[k] = (uint32_t)sa;
            } else {
                const int sb = y < lb ? (int)cmat[a * dim + rb[y]] : -128;
                w[k] = pack16x2(sa, sb);
            }
        }
        if constexpr (FORM == kPair128)
            ((uint4*)prof)[a * stride + g] = make_uint4(w[0], w[1], w[2], w[3]);
        else if constexpr (FORM == kPair32)
            ((uint32_t*)prof)[a * stride + g] = w[0];
        else if constexpr (FORM == kPair64)
            ((uint2*)prof)[a * stride + g] = make_uint2(w[0], w[1]);
        else
            ((uint2*)prof)[a * stride + g] = make_uint2(pack16x2((int)w[0], (int)w[1]), pack16x2((int)w[2], (int)w[3]));
    }
}

// The 16x2 scores of rows 4g .. 4g + 3 from the entries of the lane's residue
// (low halves; `pb`: the high halves' residue, the dual-lane form only, whose
// halves read different residues and are interleaved with byte permutes).
template <int FORM>
__device__ __forceinline__ void fetch16(const void* pa, const void* pb, int g, uint32_t (&sc)[4]) {
    if constexpr (FORM == kPair128) {
        const uint4 w = ((const uint4*)pa)[g];
        sc[0] = w.x;
        sc[1] = w.y;
        sc[2] = w.z;
        sc[3] = w.w;
    } else if constexpr (FORM == kPair32) {
#pragma unroll
        for (int k = 0; k < 4; ++k) sc[k] = ((const uint32_t*)pa)[4 * g + k];
    } else if constexpr (FORM == kPair64) {
        const uint2 u = ((const uint2*)pa)[2 * g], v = ((const uint2*)pa)[2 * g + 1];
        sc[0] = u.x;
        sc[1] = u.y;
        sc[2] = v.x;
        sc[3] = v.y;
    } else {
        const uint2 lo = ((const uint2*)pa)[g], hi = ((const uint2*)pb)[g];
        sc[0] = __byte_perm(lo.x, hi.x, 0x5410);
        sc[1] = __byte_perm(lo.x, hi.x, 0x7632);
        sc[2] = __byte_perm(lo.y, hi.y, 0x5410);
        sc[3] = __byte_perm(lo.y, hi.y, 0x7632);
    }
}

// One column of a linear strip: H of the previous column in, of this one out.
//   H = max(diag + s, left + gap, up + gap, 0)
template <int S, int FORM>
__device__ __forceinline__ void column16_linear(uint32_t (&H)[S], uint32_t diag, uint32_t up, const void* pa,
                                                const void* pb, uint32_t g2, uint32_t& mx) {
#pragma unroll
    for (int g = 0; g < S / 4; ++g) {
        uint32_t sc[4];
        fetch16<FORM>(pa, pb, g, sc);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = 4 * g + k;
            const uint32_t left = H[r];
            uint32_t h = __viaddmax_s16x2(left, g2, __vadd2(diag, sc[k]));
            h = __viaddmax_s16x2_relu(up, g2, h);
            diag = left;
            H[r] = h;
            up = h;
        }
    }
#pragma unroll
    for (int r = 0; r < S; r += 2) mx = __vimax3_s16x2(mx, H[r], H[r + 1]);
}

// One column of an affine strip.
//   M  = Bdiag + s
//   Y  = max(Yup + ext, Mg_up)      strip-axis gap chain, Mg = M + gap + ext
//   X  = Zl                         sweep-axis gap chain, computed a column ago:
//                                   Zl = max(X + ext, Mg) is the next column's X
//   B  = max(M, Y, X, 0)
// The reference floors M at 0 before the gaps open from it; a gap opened from
// a floored M is negative, as is one opened from the M below 0 here, and what
// is negative never reaches B >= 0, so every B is the same.
// In: Zl, Bl of the previous column, the first row's Y (y) and the diagonal B.
// Out: this column's; in y the Y of the row below the strip.
template <int S, int FORM>
__device__ __forceinline__ void column16_affine(uint32_t (&Zl)[S], uint32_t (&Bl)[S], uint32_t bdiag, uint32_t& y,
                                                const void* pa, const void* pb, uint32_t e2, uint32_t ge2,
                                                uint32_t& mx) {
#pragma unroll
    for (int g = 0; g < S / 4; ++g) {
        uint32_t sc[4];
        fetch16<FORM>(pa, pb, g, sc);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = 4 * g + k;
            const uint32_t m = __vadd2(bdiag, sc[k]);
            const uint32_t xg = Zl[r];
            const uint32_t bst = __vimax3_s16x2_relu(m, y, xg);
            const uint32_t mg = __vadd2(m, ge2);
            Zl[r] = __viaddmax_s16x2(xg, e2, mg);
            y = __viaddmax_s16x2(y, e2, mg);
            bdiag = Bl[r];
            Bl[r] = bst;
        }
    }
#pragma unroll
    for (int r = 0; r < S; r += 2) mx = __vimax3_s16x2(mx, Bl[r], Bl[r + 1]);
}

// ------------------------------------------------------------ chained strips
// A multi-strip item (two strip sequences against 32 lane sequences) is cut
// into one item per 32-row strip.  Strip s of a chain runs on whichever warp
// takes it, a few columns behind strip s - 1: it reads the boundary row that
// strip s - 1 writes into the chain's ring slot (two rows, alternating), as
// far as strip s - 1 has published its progress.  So one long item no longer
// runs on a single warp from its first row to its last.
//
// Ordering: the writer stores its boundary values, every lane fences
// (fence.acq_rel.gpu), the warp synchronises, and lane 0 publishes the column
// count with st.release.gpu; readers poll with ld.acquire.gpu and read the
// ring with ld.global.cg (L2, never a stale L1 line).  A ring row is
// rewritten by strip s + 2 only after strip s + 1 has published progress past
// those columns, i.e. after it has read them.
//
// Progress: entries are handed out in queue order and a strip waits only for
// its predecessor, which is queued before it and so was taken by a warp that
// is running; every wait therefore ends.  Each wait is nevertheless bounded:
// after the launch's wait limit (kChainWaitNs unless the host sets another)
// without progress, or when another warp has given up, the
// warp sets abort_flag and stops, and the host reports the launch as failed.
// Only the longest items are chained (the host plans the queue so that a
// strip is handed out about when its predecessor is kChainLead columns
// ahead); the others run whole on one warp, as in score16_kernel.
constexpr int kChainDone = 1 << 30;
// A strip publishes its progress every kChainPublish columns (one fence per
// lane each time); its successor starts once kChainLead columns are out and
// afterwards asks for kChainNeed columns beyond its current block, so that in
// the steady state it runs a publish period or more behind and its polls
// find the columns already there.
constexpr int kChainPublish = 32;
constexpr int kChainLead = 64;
constexpr int kChainNeed = 40;
// Default bound of one wait (PW_TUNE_WAIT_NS overrides it per launch).
constexpr unsigned long long kChainWaitNs = 2000000000ull;
// Boundary rows: per block of four columns and lane 16 bytes (linear: H of the
// strip's last row) or 32 (affine: B of the last row and Y of the row below
// it, which is all that the next strip needs), so that a lane stores and loads
// a block with one or two 128-bit accesses.
template <bool AFFINE>
__host__ __device__ constexpr int64_t ring_row(int xm4) { return (int64_t)(xm4 / 4) * kWarp * (AFFINE ? 2 : 1); }
// The affine sweep keeps the row above kPreBlocks - 1 column blocks in flight:
// each lane copies its own two entries into a per-warp shared-memory ring with
// cp.async (within the kChainNeed columns the chain wait guarantees); the
// linear sweep loads its one entry a block ahead into registers.
constexpr int kPreBlocks = 3;
constexpr int kPreBytes = kPreBlocks * 2 * kWarp * (int)sizeof(uint4);  // per warp
static_assert(4 * kPreBlocks <= kChainNeed, "prefetched columns must be published");

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Warp-uniform wait until *flag >= need.  Returns the smallest value the lanes
// saw (>= need), or -1 when the wait gave up after limit_ns without success or
// because another warp had given up (abort_flag is then set).
__device__ __forceinline__ int chain_wait(const int* flag, int need, int* abort_flag, unsigned long long limit_ns) {
    int v = ld_acquire_gpu(flag);
    if (__all_sync(0xffffffffu, v >= need)) return __reduce_min_sync(0xffffffffu, v);
    const unsigned long long t0 = global_ns();
    unsigned ns = 32;
    for (;;) {
        __nanosleep(ns);
        if (ns < 1024) ns <<= 1;
        v = ld_acquire_gpu(flag);
        if (__all_sync(0xffffffffu, v >= need)) return __reduce_min_sync(0xffffffffu, v);
        const bool give_up = ld_acquire_gpu(abort_flag) != 0 || global_ns() - t0 > limit_ns;
        if (__any_sync(0xffffffffu, give_up)) {
            if ((threadIdx.x & 31) == 0) atomicExch(abort_flag, 1);
            return -1;
        }
    }
}

// Publishes `v` as the item's progress after this warp's boundary stores.
__device__ __forceinline__ void chain_publish(int* flag, int v) {
    fence_acq_rel_gpu();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) st_release_gpu(flag, v);
}

// One strip of an item: a lane, two pairs (strip A / strip B against the lane
// sequence).  The column loop runs to the warp's longest lane (xm4,
// warp-uniform); a lane past its own sequence sweeps padding-code columns,
// which cannot raise its maximum (in the dual-lane form the high halves'
// second lane sequence, qc2 / lq42, likewise).  BND: the strip may have a strip
// above (has_up, its last row in row_in) and one below (has_down, row_out);
// with prog_in / prog_out they run on other warps.  Returns false when a wait
// gave up.
template <int S, bool AFFINE, int FORM, bool BND>
__device__ __forceinline__ bool sweep16(const uint8_t* qc, int lq4, const uint8_t* qc2, int lq42, int xm4,
                                        uint32_t pad4, const unsigned char* prof, int gap, int ext, bool has_up,
                                        bool has_down, const uint4* row_in, uint4* row_out, const int* prog_in,
                                        int* prog_out, int* abort_flag, unsigned long long wait_ns, uint4* pre,
                                        uint32_t& mx) {
    constexpr bool DL = FORM == kDual;
    constexpr int kResidue = prof_stride<S, FORM>() * prof_entry_bytes<FORM>();  // profile bytes a residue
    const uint32_t g2 = pack16(gap), e2 = pack16(ext), ge2 = pack16(gap + ext);
    int avail = 0;  // columns of the strip above known to be published
    auto need_cols = [&](int upto) -> bool {  // columns [0, upto) of row_in readable
        if (!BND || !prog_in || avail >= upto) return true;
        avail = chain_wait(prog_in, upto, abort_flag, wait_ns);
        return avail >= 0;
    };
    auto code_word = [&](int x4) -> uint32_t { return x4 < lq4 ? *(const uint32_t*)(qc + x4) : pad4; };
    auto code_word2 = [&](int x4) -> uint32_t { return DL && x4 < lq42 ? *(const uint32_t*)(qc2 + x4) : pad4; };
    if (!need_cols(min(kChainLead, xm4))) return false;
    // the code words of the next 4 columns and the row above's entries are
    // loaded ahead (their latency hides behind the columns' arithmetic)
    uint32_t cw_next = code_word(0), cw2_next = code_word2(0);
    uint32_t prev = 0;  // the row above, one column back: the first row's diagonal
    if constexpr (!AFFINE) {
        uint32_t H[S];
#pragma unroll
        for (int r = 0; r < S; ++r) H[r] = 0;
        uint4 in_next = BND && has_up && xm4 > 0 ? __ldcg(row_in) : make_uint4(0u, 0u, 0u, 0u);
        for (int x4 = 0; x4 < xm4; x4 += 4) {
            if (!need_cols(min(x4 + kChainNeed, xm4))) return false;
            const uint32_t cw = cw_next, cw2 = cw2_next;
            const uint4 in = in_next;
            cw_next = code_word(x4 + 4);
            if constexpr (DL) cw2_next = code_word2(x4 + 4);
            if (BND && has_up && x4 + 4 < xm4) in_next = __ldcg(row_in + (x4 / 4 + 1) * kWarp);
            uint32_t out[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const void* pa = prof + ((cw >> (8 * j)) & 0xff) * kResidue;
                const void* pb = DL ? prof + ((cw2 >> (8 * j)) & 0xff) * kResidue : pa;
                const uint32_t up = j == 0 ? in.x : j == 1 ? in.y : j == 2 ? in.z : in.w;
                column16_linear<S, FORM>(H, prev, up, pa, pb, g2, mx);
                prev = up;
                out[j] = H[S - 1];
            }
            if (BND && has_down) {
                __stcg(row_out + (x4 / 4) * kWarp, make_uint4(out[0], out[1], out[2], out[3]));
                if (prog_out && (((x4 + 4) % kChainPublish) == 0 || x4 + 4 >= xm4)) chain_publish(prog_out, x4 + 4);
            }
        }
    } else {
        // left of and above the matrix: M = 0, X and Y = -inf.
        // Zl[r] = max(X + ext, M + gap + ext) of the previous column: exactly
        // this column's X, one row array instead of two
        uint32_t Zl[S], Bl[S];
#pragma unroll
        for (int r = 0; r < S; ++r) {
            Zl[r] = ge2;
            Bl[r] = 0;
        }
        uint4* my = pre + (threadIdx.x & 31);
        auto copy_block = [&](int blk) {  // block blk's entries into slot blk % kPreBlocks
            if (4 * blk < xm4) {
                uint4* d = my + (blk % kPreBlocks) * 2 * kWarp;
                cp_async16(d, row_in + (2 * blk) * kWarp);
                cp_async16(d + kWarp, row_in + (2 * blk + 1) * kWarp);
            }
            cp_async_commit();
        };
        if (BND && has_up) {
#pragma unroll
            for (int k = 0; k < kPreBlocks - 1; ++k) copy_block(k);
        }
        for (int x4 = 0; x4 < xm4; x4 += 4) {
            if (!need_cols(min(x4 + kChainNeed, xm4))) {
                cp_async_wait<0>();  // no copy outlives the sweep
                return false;
            }
            const uint32_t cw = cw_next, cw2 = cw2_next;
            cw_next = code_word(x4 + 4);
            if constexpr (DL) cw2_next = code_word2(x4 + 4);
            uint4 in0 = make_uint4(kNeg16x2, 0u, kNeg16x2, 0u), in1 = in0;
            if (BND && has_up) {
                copy_block(x4 / 4 + kPreBlocks - 1);  // its slot held the block before this one
                cp_async_wait<kPreBlocks - 1>();      // this block's copies have landed
                const uint4* d = my + ((x4 / 4) % kPreBlocks) * 2 * kWarp;
                in0 = d[0];
                in1 = d[kWarp];
            }
            uint4 out0, out1;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const void* pa = prof + ((cw >> (8 * j)) & 0xff) * kResidue;
                const void* pb = DL ? prof + ((cw2 >> (8 * j)) & 0xff) * kResidue : pa;
                uint32_t y = j == 0 ? in0.x : j == 1 ? in0.z : j == 2 ? in1.x : in1.z;
                column16_affine<S, FORM>(Zl, Bl, prev, y, pa, pb, e2, ge2, mx);
                prev = j == 0 ? in0.y : j == 1 ? in0.w : j == 2 ? in1.y : in1.w;
                if (j == 0) out0.x = y, out0.y = Bl[S - 1];
                if (j == 1) out0.z = y, out0.w = Bl[S - 1];
                if (j == 2) out1.x = y, out1.y = Bl[S - 1];
                if (j == 3) out1.z = y, out1.w = Bl[S - 1];
            }
            if (BND && has_down) {
                uint4* d = row_out + (x4 / 2) * kWarp;
                __stcg(d, out0);
                __stcg(d + kWarp, out1);
                if (prog_out && (((x4 + 4) % kChainPublish) == 0 || x4 + 4 >= xm4)) chain_publish(prog_out, x4 + 4);
            }
        }
        if constexpr (BND) cp_async_wait<0>();
    }
    return true;
}

// One item's lanes.  Strip-pair form: strip A (W.target) in the low halves,
// strip B (W.index, or none) in the high halves, one lane sequence per lane.
// Dual-lane form (DL): strip W.target in both halves, the lane sequences of
// sorted positions W.first + lane (low) and W.first + 32 + lane (high, the
// first W.lanes_hi lanes).
struct Lanes16 {
    bool active;        // the low half's lane sequence exists
    int p, p2;          // lane sequences of the low / high halves
    const uint8_t* qc;  // their codes
    const uint8_t* qc2;
    int lq4, lq42;      // their lengths rounded up to 4 (0: padding only)
};

template <bool DL>
__device__ __forceinline__ Lanes16 item_lanes(const Score16Args& A, const WorkItem& W, int lane) {
    Lanes16 L;
    L.active = lane < W.lanes;
    L.p = L.active ? A.lane_order[W.first + lane] : 0;
    L.qc = A.lane_codes + A.lane_off[L.p];
    L.lq4 = L.active ? (A.lane_len[L.p] + 3) & ~3 : 0;
    const bool hi = DL && lane < W.lanes_hi;
    L.p2 = hi ? A.lane_order[W.first + kWarp + lane] : -1;
    L.qc2 = hi ? A.lane_codes + A.lane_off[L.p2] : L.qc;
    L.lq42 = hi ? (A.lane_len[L.p2] + 3) & ~3 : 0;
    return L;
}

// Work item `it` of a grid-form launch (see Score16Args::grid_strips).
template <int S, bool DL>
__device__ __forceinline__ WorkItem grid_item(const Score16Args& A, int it) {
    const int g = it / A.grid_n_strips, p = it - g * A.grid_n_strips;
    const int2 sp = A.grid_strips[p];
    WorkItem W;
    W.target = sp.x;
    W.index = sp.y;
    W.first = g * A.grid_lane_step;
    W.lanes = min(kWarp, A.grid_n_lane - W.first);
    W.lanes_hi = DL ? max(0, min(kWarp, A.grid_n_lane - W.first - kWarp)) : 0;
    W.xmax = A.lane_len[A.lane_order[W.first]];
    W.S = S;
    W.orient = 0;
    W.dir_base = 0;
    W.pair_base = 0;
    return W;
}

// Writes a lane's two pair maxima (NaN where the 16-bit limit was reached).
template <bool DL>
__device__ __forceinline__ void store_max16(const Score16Args& A, const WorkItem& W, const Lanes16& L, uint32_t mx) {
    const int sa = W.target;
    const int s_hi = DL ? (L.p2 >= 0 ? sa : -1) : W.index;
    const int p_hi = DL ? L.p2 : L.p;
    const int ma = (int)(int16_t)(mx & 0xffffu), mb = (int)(int16_t)(mx >> 16);
    A.pair_max[(int64_t)sa * A.stride_strip + (int64_t)L.p * A.stride_lane] =
        ma >= kOvf16 ? __int_as_float(0x7fc00000) : (float)ma;
    if (s_hi >= 0)
        A.pair_max[(int64_t)s_hi * A.stride_strip + (int64_t)p_hi * A.stride_lane] =
            mb >= kOvf16 ? __int_as_float(0x7fc00000) : (float)mb;
    if (ma >= kOvf16 || (s_hi >= 0 && mb >= kOvf16)) atomicAdd(A.ovf_count, 1);
}

// A block's shared memory: its four warps' profiles, then (affine, with
// boundary rows) their prefetch rings.
template <int S, bool AFFINE, int FORM, bool BND>
__host__ __device__ constexpr int score16_smem(int alpha1) {
    return block_profile_bytes<S, FORM>(alpha1) + (AFFINE && BND ? 4 * kPreBytes : 0);
}

// Every strip of an item on this warp, its boundary rows in the warp's slot of
// bnd_pool.
template <int S, bool AFFINE, int FORM, bool MULTI>
__device__ __forceinline__ uint32_t whole_item16(const Score16Args& A, const WorkItem& W, const Lanes16& L,
                                                 unsigned char* prof, uint4* pre, uint4* bnd, int lane) {
    const int sa = W.target, sb = FORM == kDual ? -1 : W.index;
    const int la = A.strip_len[sa];
    const int lb = sb >= 0 ? A.strip_len[sb] : 0;
    const uint8_t* ra = A.strip_res + A.strip_off[sa];
    const uint8_t* rb = A.strip_res + A.strip_off[sb >= 0 ? sb : sa];
    const int nstrips = MULTI ? (max(la, lb) + S - 1) / S : 1;
    const int xm4 = (W.xmax + 3) & ~3;
    const int64_t row = ring_row<AFFINE>(xm4);
    const uint32_t pad4 = (uint32_t)A.pad_code * 0x01010101u;
    uint32_t mx = 0;
    for (int st = 0; st < nstrips; ++st) {
        if (MULTI && st > 0) fence_acq_rel_gpu();  // the row above is stored before it is copied back
        __syncwarp();
        build_profile16<S, FORM>(prof, A.cmat, ra, rb, st * S, la, lb, A.alpha1, A.dim, lane);
        __syncwarp();
        const uint4* row_in = MULTI ? bnd + ((st + 1) & 1) * row : nullptr;
        uint4* row_out = MULTI ? bnd + (st & 1) * row : nullptr;
        sweep16<S, AFFINE, FORM, MULTI>(L.qc, L.lq4, L.qc2, L.lq42, xm4, pad4, prof, A.gap, A.ext, st > 0,
                                        st + 1 < nstrips, row_in, row_out, nullptr, nullptr, nullptr, 0ull, pre, mx);
    }
    return mx;
}

template <int S, bool AFFINE, int FORM>
__global__ void __launch_bounds__(128, AFFINE ? 3 : 4) score16_chain_kernel(Score16Args A) {
    constexpr bool DL = FORM == kDual;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    unsigned char* prof = smem + wib * warp_profile_bytes<S, FORM>(A.alpha1);
    uint4* pre = (uint4*)(smem + block_profile_bytes<S, FORM>(A.alpha1) + wib * kPreBytes);
    const uint32_t pad4 = (uint32_t)A.pad_code * 0x01010101u;
    const int64_t warp_global = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    for (;;) {
        int it = 0;
        if (lane == 0) it = A.item_base + atomicAdd(A.counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= A.n_items) break;
        const int4 ci = A.chain[it];
        const WorkItem W = A.items[ci.w];
        const int c = ci.x, pred = ci.z;
        const bool whole = ci.y < 0;
        const int sa = W.target, sb = DL ? -1 : W.index;
        const int la = A.strip_len[sa];
        const int lb = sb >= 0 ? A.strip_len[sb] : 0;
        const int nstrips = (max(la, lb) + S - 1) / S;
        const Lanes16 L = item_lanes<DL>(A, W, lane);
        const uint8_t* ra = A.strip_res + A.strip_off[sa];
        const uint8_t* rb = A.strip_res + A.strip_off[sb >= 0 ? sb : sa];
        const int xm4 = (W.xmax + 3) & ~3;
        const int64_t row = ring_row<AFFINE>(xm4);
        uint4* rows = (whole ? A.bnd_pool + warp_global * A.bnd_slot : A.ring + A.ring_off[c]) + lane;
        // a chain entry is one strip; a whole item runs its strips one after
        // another here, without progress flags
        uint32_t mx = 0;
        bool ok = true;
        int s = whole ? 0 : ci.y;
        const int s_end = whole ? nstrips : s + 1;
        for (; s < s_end && ok; ++s) {
            if (whole && s > 0) fence_acq_rel_gpu();  // the row above is stored before it is copied back
            __syncwarp();
            build_profile16<S, FORM>(prof, A.cmat, ra, rb, s * S, la, lb, A.alpha1, A.dim, lane);
            __syncwarp();
            const bool has_down = s + 1 < nstrips;
            ok = sweep16<S, AFFINE, FORM, true>(L.qc, L.lq4, L.qc2, L.lq42, xm4, pad4, prof, A.gap, A.ext, s > 0,
                                                has_down, rows + ((s + 1) & 1) * row, rows + (s & 1) * row,
                                                !whole && s > 0 ? A.progress + pred : nullptr,
                                                !whole && has_down ? A.progress + it : nullptr, A.abort_flag,
                                                A.wait_ns, pre, mx);
        }
        if (!ok) break;
        bool finished = true;
        if (!whole) {
            if (ci.y > 0) {
                // the predecessor's running maximum is final once it has finished
                if (chain_wait(A.progress + pred, kChainDone, A.abort_flag, A.wait_ns) < 0) break;
                mx = __vmaxs2(mx, __ldcg(&A.run_max[(int64_t)pred * kWarp + lane]));
            }
            if (ci.y + 1 < nstrips) {
                __stcg(&A.run_max[(int64_t)it * kWarp + lane], mx);
                chain_publish(A.progress + it, kChainDone);
                finished = false;
            }
        }
        if (finished && L.active) store_max16<DL>(A, W, L, mx);
    }
}

template <int S, bool AFFINE, bool MULTI, int FORM>
__global__ void __launch_bounds__(128) score16_kernel(Score16Args A) {
    constexpr bool DL = FORM == kDual;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    unsigned char* prof = smem + wib * warp_profile_bytes<S, FORM>(A.alpha1);
    uint4* pre = (uint4*)(smem + block_profile_bytes<S, FORM>(A.alpha1) + wib * kPreBytes);
    const int64_t warp_global = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    uint4* bnd = MULTI ? A.bnd_pool + warp_global * A.bnd_slot + lane : nullptr;
    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(A.counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= A.n_items) break;
        const WorkItem W = A.grid_strips ? grid_item<S, DL>(A, it) : A.items[it];
        const Lanes16 L = item_lanes<DL>(A, W, lane);
        const uint32_t mx = whole_item16<S, AFFINE, FORM, MULTI>(A, W, L, prof, MULTI ? pre : nullptr, bnd, lane);
        if (L.active) store_max16<DL>(A, W, L, mx);
    }
}

}  // namespace pw

// pw_finish.cuh -- hit order and alignment strings on the device.
//
// The walk leaves its hits (DevHit) and their column operations ('M', 'I',
// 'D' per alignment column) in device memory, appended across memory waves.
// These kernels put the hits in the order the reference's HitList has them
// and spell out the three alignment strings of every hit, so that the host
// receives the final records in two copies.
//
// Order (SmithWaterman._print_alignments appends in the pinned emission
// order of the starting points and HitList sorts by score,
// SmithWaterman.py:699): score ascending; then block anti-diagonal
// descending, block x descending, target, query, cell anti-diagonal
// descending, row ascending; then walk order.  The key's fields are packed into
// one 64-bit word of as many bits as the inputs need (HitKeyBits; scores are >=
// 0, so integer scores order as integers and fp32 ones by their bits): up to
// kSmallHits hits are ranked by one block, more by one stable radix sort of
// those bits (1.1 million hits of 150-residue reads: 50 bits; three sorts of 64
// bits took 0.6 ms longer).  Keys that need more than 64 bits are split into
// three words and sorted by three stable passes, least significant word first.
#pragma once
#include "../../include/paswas_b200.h"
#include "pw_device.cuh"

namespace pw {

__global__ void hit_key_kernel(const DevHit* h, int64_t n, uint64_t* ka, uint64_t* kb, uint64_t* kc, int32_t* idx) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const DevHit d = h[k];
        const uint32_t sb = __float_as_uint(d.score);
        const uint32_t diag = (uint32_t)((d.end_x >> 3) + (d.end_y >> 3));
        const uint32_t small = (uint32_t)((d.end_x & 7) + (d.end_y & 7));
        ka[k] = ((uint64_t)sb << 32) | (0xFFFFFFFFu - diag);
        kb[k] = ((uint64_t)(0xFFFFFFFFu - (uint32_t)(d.end_x >> 3)) << 32) | (uint32_t)d.target;
        kc[k] = ((uint64_t)(uint32_t)d.query << 32) | ((uint64_t)(0xFFu - small) << 8) | (uint32_t)(d.end_y & 7);
        idx[k] = (int32_t)k;
    }
}

__global__ void gather_key_kernel(const uint64_t* src, const int32_t* idx, int64_t n, uint64_t* dst) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        dst[k] = src[idx[k]];
}

// Field widths of the packed key, most significant field first: score, block
// anti-diagonal (descending from diag_top), block x (descending from x_top),
// target, query, cell anti-diagonal (4 bits, descending), row (3 bits).
struct HitKeyBits {
    int diag, x, target, query;
    uint32_t diag_top, x_top;
    int is_float;
};

__device__ __forceinline__ uint64_t packed_key(const DevHit& d, const HitKeyBits& B) {
    const uint32_t bx = (uint32_t)(d.end_x >> 3), by = (uint32_t)(d.end_y >> 3);
    const uint32_t small = (uint32_t)((d.end_x & 7) + (d.end_y & 7));
    uint64_t k = B.is_float ? __float_as_uint(d.score) : (uint32_t)d.score;
    k = k << B.diag | (B.diag_top - (bx + by));
    k = k << B.x | (B.x_top - bx);
    k = k << B.target | (uint32_t)d.target;
    k = k << B.query | (uint32_t)d.query;
    return k << 7 | (uint64_t)(14u - small) << 3 | (uint32_t)(d.end_y & 7);
}

__global__ void hit_pack_kernel(const DevHit* h, int64_t n, HitKeyBits B, uint64_t* key, int32_t* idx) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        key[k] = packed_key(h[k], B);
        idx[k] = (int32_t)k;
    }
}

// Up to kSmallHits hits in one block: each thread ranks its hit among all of
// them (keys in shared memory, ties by walk order), then the string lengths in
// order and their exclusive scan.
constexpr int kSmallHits = 1024;
__global__ void __launch_bounds__(kSmallHits) hit_small_kernel(const DevHit* h, int n, HitKeyBits B, int32_t* idx,
                                                               int64_t* len, int64_t* soff) {
    __shared__ uint64_t key[kSmallHits];
    __shared__ int32_t cols[kSmallHits];
    __shared__ int64_t part[32];
    const int k = threadIdx.x, lane = k & 31;
    uint64_t mine = 0;
    if (k < n) key[k] = mine = packed_key(h[k], B);
    __syncthreads();
    int rank = 0;
    if (k < n) {
        for (int j = 0; j < n; ++j) rank += (key[j] < mine || (key[j] == mine && j < k)) ? 1 : 0;
        idx[rank] = k;
        cols[rank] = h[k].n_cols;
    }
    __syncthreads();
    const int64_t bytes = k < n ? 3 * (int64_t)cols[k] : 0;
    int64_t sum = bytes;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    if (lane == 31) part[k >> 5] = sum;
    __syncthreads();
    int64_t before = 0;
    for (int w = 0; w < (k >> 5); ++w) before += part[w];
    if (k < n) {
        len[k] = bytes;
        soff[k] = before + sum - bytes;
    }
}

// String bytes of the hit at each sorted position (three strings of n_cols).
__global__ void hit_len_kernel(const DevHit* h, const int32_t* idx, int64_t n, int64_t* len) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        len[k] = 3 * (int64_t)h[idx[k]].n_cols;
}

// The hit records in order and their strings: sequence_match (query residue
// or '-'), alignment ('|' for equal residues -- letters compared without
// case -- '.' for a mismatch, ' ' in a gap) and target_match, one column per
// operation, as SmithWaterman._print_alignments spells them
// (SmithWaterman.py:765-815).
// A thread spells hits of up to kWarpStringCols columns here; longer ones get
// only their record, a warp spells them up to kBlockStringCols columns
// (hit_strings_warp_kernel) and a block beyond (hit_strings_block_kernel: a 25
// kb hit took a warp 3.2 ms).
constexpr int kWarpStringCols = 32;
constexpr int kBlockStringCols = 2048;

// One column's characters: operation c, query position px, target position py.
__device__ __forceinline__ void spell_column(char c, const uint8_t* qs, const uint8_t* ts, int px, int py, char* sq,
                                             char* al, char* tg, int i) {
    if (c == 'M') {
        const uint8_t ca = ts[py], cb = qs[px];
        const bool la = (ca >= 'A' && ca <= 'Z') || (ca >= 'a' && ca <= 'z');
        const bool eq = la ? ((ca | 0x20) == (cb | 0x20)) : ca == cb;
        sq[i] = (char)cb;
        tg[i] = (char)ca;
        al[i] = eq ? '|' : '.';
    } else if (c == 'I') {
        sq[i] = (char)qs[px];
        tg[i] = '-';
        al[i] = ' ';
    } else {
        sq[i] = '-';
        tg[i] = (char)ts[py];
        al[i] = ' ';
    }
}

__global__ void hit_out_kernel(const DevHit* h, const int32_t* idx, const int64_t* soff, int64_t n, const char* ops,
                               const uint8_t* q_raw, const int64_t* q_off, const uint8_t* t_raw,
                               const int64_t* t_off, pw_hit* out, char* str) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const DevHit d = h[idx[k]];
        pw_hit o;
        o.query = d.query;
        o.target = d.target;
        o.s_start = d.s_start;
        o.s_end = d.s_end;
        o.t_start = d.t_start;
        o.t_end = d.t_end;
        o.score = d.score;
        o.matches = d.matches;
        o.mismatches = d.mismatches;
        o.n_cols = d.n_cols;
        o.str_offset = soff[k];
        out[k] = o;
        if (d.n_cols > kWarpStringCols) continue;
        char* sq = str + o.str_offset;
        char* al = sq + d.n_cols;
        char* tg = al + d.n_cols;
        const uint8_t* qs = q_raw + q_off[d.query];
        const uint8_t* ts = t_raw + t_off[d.target];
        const char* op = ops + d.ops_offset;
        int x = d.s_start, y = d.t_start;
        for (int i = 0; i < d.n_cols; ++i) {
            const char c = op[i];
            spell_column(c, qs, ts, x, y, sq, al, tg, i);
            x += c != 'D' ? 1 : 0;
            y += c != 'I' ? 1 : 0;
        }
    }
}

// The strings of the longer hits, one warp per hit and 32 columns per step:
// the query / target position of every column is the starting position plus
// the number of earlier columns that consume a query residue ('M', 'I') or a
// target residue ('M', 'D').  A warp takes `group` consecutive hits (lengths
// read together) and spells those in its range of lengths.
__global__ void hit_strings_warp_kernel(const DevHit* h, const int32_t* idx, const int64_t* soff, const int64_t* len,
                                        int64_t n, int group, const char* ops, const uint8_t* q_raw,
                                        const int64_t* q_off, const uint8_t* t_raw, const int64_t* t_off, char* str) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t k0 = warp * group; k0 < n; k0 += warps * group) {
        const int64_t mine = lane < group && k0 + lane < n ? len[k0 + lane] / 3 : 0;
        unsigned todo = __ballot_sync(0xffffffffu, mine > kWarpStringCols && mine <= kBlockStringCols);
        while (todo) {
            const int64_t k = k0 + __ffs(todo) - 1;
            todo &= todo - 1;
            const DevHit d = h[idx[k]];
            char* sq = str + soff[k];
            const uint8_t* qs = q_raw + q_off[d.query];
            const uint8_t* ts = t_raw + t_off[d.target];
            const char* op = ops + d.ops_offset;
            int x = d.s_start, y = d.t_start;
            for (int c0 = 0; c0 < d.n_cols; c0 += 32) {
                const int i = c0 + lane;
                const bool act = i < d.n_cols;
                const char c = act ? op[i] : 'M';
                const unsigned mx = __ballot_sync(0xffffffffu, act && c != 'D');
                const unsigned my = __ballot_sync(0xffffffffu, act && c != 'I');
                if (act)
                    spell_column(c, qs, ts, x + __popc(mx & below), y + __popc(my & below), sq, sq + d.n_cols,
                                 sq + 2 * (int64_t)d.n_cols, i);
                x += __popc(mx);
                y += __popc(my);
            }
        }
    }
}

// The strings of the longest hits, one block per hit and blockDim.x columns
// per step.
__global__ void __launch_bounds__(512) hit_strings_block_kernel(const DevHit* h, const int32_t* idx,
                                                                const int64_t* soff, const int64_t* len, int64_t n,
                                                                const char* ops, const uint8_t* q_raw,
                                                                const int64_t* q_off, const uint8_t* t_raw,
                                                                const int64_t* t_off, char* str) {
    __shared__ int cx[2][16], cy[2][16];  // per warp: consuming columns of this step
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    int flip = 0;
    for (int64_t k = blockIdx.x; k < n; k += gridDim.x) {
        if (len[k] / 3 <= kBlockStringCols) continue;
        const DevHit d = h[idx[k]];
        char* sq = str + soff[k];
        const uint8_t* qs = q_raw + q_off[d.query];
        const uint8_t* ts = t_raw + t_off[d.target];
        const char* op = ops + d.ops_offset;
        int x = d.s_start, y = d.t_start;
        for (int c0 = 0; c0 < d.n_cols; c0 += 512) {
            const int i = c0 + (int)threadIdx.x;
            const bool act = i < d.n_cols;
            const char c = act ? op[i] : 'M';
            const unsigned mx = __ballot_sync(0xffffffffu, act && c != 'D');
            const unsigned my = __ballot_sync(0xffffffffu, act && c != 'I');
            if (lane == 0) {
                cx[flip][wib] = __popc(mx);
                cy[flip][wib] = __popc(my);
            }
            __syncthreads();
            int px = x + __popc(mx & below), py = y + __popc(my & below);
#pragma unroll
            for (int w = 0; w < 16; ++w) {
                const int vx = cx[flip][w], vy = cy[flip][w];
                if (w < wib) {
                    px += vx;
                    py += vy;
                }
                x += vx;
                y += vy;
            }
            flip ^= 1;  // the other buffer is free: every warp has passed this step's barrier
            if (act) spell_column(c, qs, ts, px, py, sq, sq + d.n_cols, sq + 2 * (int64_t)d.n_cols, i);
        }
    }
}

}  // namespace pw

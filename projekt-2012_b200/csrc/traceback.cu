// traceback.cu -- stage 2: the alignment (canonical traceback) on the GPU.
//
// Replaces the reference's stage 2 (src/Crosspointer.cpp:104-338 with the
// reverse kernels of src/TraceBack.cuh:7-472 and the host join of
// src/SWutils.cpp:175-231).  The reference searches backwards for crosspoints
// on its special rows; its search hangs or exits on most inputs, so this library
// defines the path directly: the traceback of the forward matrix from the end
// cell with a fixed precedence (in H: diagonal > E (column base against a gap)
// > F (row base against a gap); in E or F: extend > open), and reports the
// reference's crosspoints (the path's last cell on every row X with
// (X + 1) % (4T) == 0, src/Builders.cpp:16) along that path.  The path does not
// depend on any tuning parameter of this library.
//
// How: stage 1 keeps special rows (H, F) at every strip bottom (every 448 or 512
// rows, the strip height) and special columns (H, E) every 256 columns, so every
// block of that grid (at most 512 x 256) can be recomputed from its stored
// boundaries alone, with four direction bits per cell.
// A block's directions do not depend on the path, so the walker of a single
// pair (walk_region) recomputes a predicted corridor of whole blocks at once,
// one CTA per block across the GPU (the staircase of blocks along the diagonal
// from the current cell, with the blocks above and to the left as margin), and
// then one warp walks the path through them (32 cells per ballot along
// diagonal, row or column runs) until it reaches the start or leaves the
// corridor, where the next round predicts from.  Before that, a pair of many
// blocks is cut into segments at special rows: one CTA per segment guesses the
// cell where the path crosses its lower row (the row's best H near the diagonal)
// and walks from there on blocks it recomputes on demand; a chain of segments
// whose ends meet is the path, whatever was guessed.  Batches of pairs use one CTA
// per pair or segment.  Inside a CTA the
// block recompute is a pipeline of two warps of 256 rows each in packed 16-bit
// halves (four of 128 rows in 32 bits for scoring too wide for them), handing rows
// down through shared memory with tagged 64-bit words instead of barriers.
// Pairs whose stores would not fit the HBM budget keep a coarser grid (level 1);
// each level-1 cell near the expected path is recomputed by the batched scoring
// kernel on that sub-rectangle, which writes the 512 x 256 stores for it (level 2),
// and the corridors of blocks run across the cells.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "batch.h"
#include "traceback.h"

namespace swb {
namespace tb {

namespace {

constexpr int kBR = 512;          // block rows (= stage-1 strip height at R = 16)
constexpr int kBC = 256;          // block columns (= special-column spacing)
constexpr int kRW = 4;            // rows per recompute half lane
constexpr int kWarpRows = 64 * kRW;          // rows of a recompute warp (64 virtual lanes)
constexpr int kThreads = kBR / kWarpRows * 32;  // packed recompute threads (two warps)
constexpr int kThreadsWide = kBR / kRW;      // 32-bit recompute threads (one per four rows)

// Direction bits of a cell (a nibble).  H comes from the diagonal unless ND is set,
// then from E unless NE is set, then from F; E and F extend unless NEX / NFX is
// set.  A cell with H = 0 is on no path: the walk knows the path's prefix score
// and stops at the cell whose diagonal predecessor has none left.
enum : uint32_t { BIT_ND = 1, BIT_NE = 2, BIT_NEX = 4, BIT_NFX = 8 };
enum : int32_t { ST_H = 0, ST_E = 1, ST_F = 2 };

struct WalkArgs {
    const uint8_t *rows, *cols;
    int64_t m, n;                  // whole matrix
    int32_t match, mismatch, open, ext;
    int32_t score;                 // best score (start of the suffix accounting)
    // stores of the current region: rows [rr0, m) x cols [cc0, n) relative
    const int2 *srows;             // [q][ncols_region] (H, F) of region row (q+1)*512 - 1
    const int2 *scols;             // [q][nrows_region] (H, E) of region col (q+1)*256 - 1
    int64_t rr0, cc0;              // region origin
    int64_t rr1, cc1;              // region end (exclusive) for store indexing
    const int2 *rtop;              // (H, F) of row rr0 - 1 over region cols (nullptr: zero)
    const int2 *rleft;             // (H, E) of col cc0 - 1 over region rows (nullptr: zero)
    int32_t xp_interval;           // reference special-row spacing (4T)
    char *ops;                     // reversed op stream (end -> start)
    int64_t ops_cap;
    int64_t *xps;                  // reversed crosspoints: 4 int64 each (row, col, score, gap)
    int64_t xp_cap;
    int64_t *st;                   // walker state in/out: see kSt* below
    int32_t br;                    // block rows of the region's grid (the special-row spacing), <= kBR
    int32_t wide;                  // recompute in 32 bits (walk16_fits does not hold)
};

// walker state slots
enum { kStR = 0, kStC, kStState, kStNOps, kStSuffix, kStNXp, kStDone, kStErr, kStStartR, kStStartC, kStN };

// H, E, F of the boundary cells around a block (region-relative fetches).
__device__ __forceinline__ int2 top_hf(const WalkArgs &a, int64_t R0, int64_t c) {
    // (H, F) of row R0 - 1 at column c (c >= cc0 - 1 handled by callers)
    if (R0 == 0) return make_int2(0, 0);
    if (R0 == a.rr0) {
        if (c < a.cc0) return make_int2((a.rtop && a.rleft) ? a.rtop[-1].x : 0, 0);  // the corner
        return a.rtop ? a.rtop[c - a.cc0] : make_int2(0, 0);
    }
    const int64_t q = (int32_t)(R0 - a.rr0) / a.br - 1;
    if (c < a.cc0) return make_int2(a.rleft ? a.rleft[R0 - 1 - a.rr0].x : 0, 0);
    return a.srows[q * (a.cc1 - a.cc0) + (c - a.cc0)];
}
__device__ __forceinline__ int2 left_he(const WalkArgs &a, int64_t C0, int64_t r) {
    // (H, E) of column C0 - 1 at row r >= rr0
    if (C0 == 0) return make_int2(0, 0);
    if (C0 == a.cc0) return a.rleft ? a.rleft[r - a.rr0] : make_int2(0, 0);
    const int64_t q = (C0 - a.cc0) / kBC - 1;
    return a.scols[q * (a.rr1 - a.rr0) + (r - a.rr0)];
}

// Block inputs staged in shared memory before a recompute, so that the step loop
// and the walk touch no global memory: the top boundary (H, F) of row R0 - 1 at
// columns C0 - 1 .. C1 (index j + 1), and the row / column bytes of the block.
struct Stage {
    int2 top[kBC + 1];
    uint8_t rb[kBR];
    uint8_t cb[kBC];
    uint32_t top16[kBC + 8];       // packed recompute: H | F << 16 of row R0 - 1, offsets from base
    uint16_t col16[64 + kBC + 72]; // packed recompute: column codes, 64 entries of slack in front
};

// Loads a thread issues together (one at a time they were a chain of global round
// trips, a sixth of a block's recompute).
constexpr int kStageBatch = 4;
__device__ void stage_block(const WalkArgs &a, int64_t R0, int64_t R1, int64_t C0, int64_t C1, Stage *s) {
    const int w = (int)(C1 - C0 + 1), h = (int)(R1 - R0 + 1), nt = (int)blockDim.x;
    for (int j0 = (int)threadIdx.x - 1; j0 < w; j0 += kStageBatch * nt) {
        int2 t[kStageBatch];
        uint8_t b[kStageBatch];
#pragma unroll
        for (int q = 0; q < kStageBatch; ++q) {
            const int j = j0 + q * nt;
            if (j < w) {
                t[q] = top_hf(a, R0, C0 + j);
                b[q] = j >= 0 ? a.cols[C0 + j] : 0;
            }
        }
#pragma unroll
        for (int q = 0; q < kStageBatch; ++q) {
            const int j = j0 + q * nt;
            if (j < w) {
                s->top[j + 1] = t[q];
                if (j >= 0) {
                    s->cb[j] = b[q];
                    s->col16[64 + j] = (uint16_t)((uint32_t)b[q] << 6);
                }
            }
        }
    }
    for (int i0 = (int)threadIdx.x; i0 < h; i0 += 2 * kStageBatch * nt) {
        uint8_t b[2 * kStageBatch];
#pragma unroll
        for (int q = 0; q < 2 * kStageBatch; ++q)
            if (i0 + q * nt < h) b[q] = a.rows[R0 + i0 + q * nt];
#pragma unroll
        for (int q = 0; q < 2 * kStageBatch; ++q)
            if (i0 + q * nt < h) s->rb[i0 + q * nt] = b[q];
    }
}

// Direction nibbles of one block, in the recompute's step order so that every warp
// store is one coalesced 128-byte line: word (warp, k, lane) holds rows 4v .. 4v + 3
// of column k - v for the virtual lanes v = lane (low half) and lane + 32 (high
// half) of the warp's 256 rows.
constexpr int kC = 8;  // recompute steps between refills
constexpr int kSteps = (kBC + 63 + kC - 1) / kC * kC;
constexpr int64_t kBlockWords = (int64_t)(kBR / kWarpRows) * kSteps * 32;
__device__ __forceinline__ int dir_index(int i, int j) {  // of the 16-bit half that holds row i, column j
    const int v = (i >> 2) & 63, warp = i >> 8;
    return ((warp * kSteps + j + v) * 32 + (v & 31)) * 2 + (v >> 5);
}
struct Dir {
    const uint32_t *d;  // global or shared memory
    __device__ __forceinline__ uint32_t at(int64_t i, int64_t j) const {
        return (uint32_t)reinterpret_cast<const uint16_t *>(d)[dir_index((int)i, (int)j)] >> (4 * (i & 3));
    }
};
constexpr size_t kDirTileBytes = sizeof(uint32_t) * (size_t)kBlockWords;  // 81,920: a multiple of 16

// Hand-off between the warps of a recompute, column by column, as 64-bit words
// {value, gen}, gen being the recompute's generation; the reader re-reads until the
// tag shows the current generation.  A 64-bit shared access is single-copy atomic,
// so the tag proves its value is current without any fence.  Packed recompute:
// one boundary, H | F << 16 as offsets; 32-bit recompute: three, H and F apart.
struct Xchg {
    unsigned long long bnd[kThreadsWide / 32 - 1][kBC][2];
    int32_t err;
    uint32_t gen;  // generations used so far by this CTA (tags start at 1; entries start at 0)
};

// Zeroes the hand-off tags and the generation count (once per CTA).
__device__ void xchg_init(Xchg *x) {
    unsigned long long *p = &x->bnd[0][0][0];
    for (int i = threadIdx.x; i < (kThreadsWide / 32 - 1) * kBC * 2; i += blockDim.x) p[i] = 0ULL;
    if (threadIdx.x == 0) {
        x->err = 0;
        x->gen = 0;
    }
}

// Upper bound of a warp's wait for the warp above (SM cycles, about 1 s); the
// writer is a warp of the same CTA, so this only guards against a defect.
constexpr long long kXchgWaitCycles = 2LL * 1000 * 1000 * 1000;

__device__ __forceinline__ unsigned long long pack(uint32_t v, uint32_t gen) {
    return ((unsigned long long)gen << 32) | v;
}
__device__ __forceinline__ unsigned long long ld_shared_volatile(const unsigned long long *p) {
    return *reinterpret_cast<const volatile unsigned long long *>(p);
}

// Waits until *p carries generation gen and returns its value.  After one wait ran
// out (x->err set) it no longer waits: the warp finishes its loop on whatever
// values it reads and the caller discards the block.
__device__ __forceinline__ uint32_t take(Xchg *x, const unsigned long long *p, uint32_t gen, bool &fail) {
    unsigned long long v = ld_shared_volatile(p);
    if ((uint32_t)(v >> 32) != gen && !fail) {
        const long long t0 = clock64();
        for (;;) {
            v = ld_shared_volatile(p);
            if ((uint32_t)(v >> 32) == gen) break;
            if (clock64() - t0 > kXchgWaitCycles) {
                fail = true;
                x->err = 1;
                break;
            }
        }
    }
    return (uint32_t)v;
}

// Recomputes block rows [R0, R1] x cols [C0, C1] into d in 32 bits.  Expects
// stage_block() to have filled `s`, x->err zeroed, and a barrier after both; `gen`
// must differ from every earlier recompute of this CTA.  Thread t owns rows
// R0 + 4t .. R0 + 4t + 3: each warp is a 128-row wavefront (lane l computes column
// k - l at step k, rows passed down by shuffles) and the four warps form a pipeline
// through x, so no CTA barrier is needed inside the column loop.  For scoring whose
// values do not fit 16 bits over a block.
__device__ void recompute_wide(const WalkArgs &a, int64_t R0, int64_t R1, int64_t C0, int64_t C1, uint32_t *d, Xchg *x,
                               const Stage *s, uint32_t gen) {
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const int64_t w = C1 - C0 + 1;
    const int64_t r0 = R0 + (int64_t)t * kRW;  // my first row
    if (R0 + (int64_t)warp * 32 * kRW > R1) return;  // this warp (and every warp below it) has no rows
    int32_t Hl[kRW], El[kRW];
    uint8_t ra[kRW];
#pragma unroll
    for (int i = 0; i < kRW; ++i) {
        const int64_t r = r0 + i;
        if (r <= R1) {
            const int2 v = left_he(a, C0, r);
            Hl[i] = v.x;
            El[i] = v.y;
            ra[i] = s->rb[r - R0];
        } else {
            Hl[i] = 0;
            El[i] = 0;
            ra[i] = 0;
        }
    }
    // H of the row above my first row at column C0 - 1
    int32_t hdiag0;
    if (t == 0) hdiag0 = s->top[0].x;
    else hdiag0 = (r0 - 1 <= R1) ? left_he(a, C0, r0 - 1).x : 0;
    bool fail = false;
    __syncwarp();
    int32_t upH = 0, upF = 0;  // (H, F) from the row above at my current column
    int32_t prevUpH = hdiag0;  // H of the row above at the previous column
    const bool publish = (lane == 31) && warp < kThreadsWide / 32 - 1 && (r0 + kRW - 1 <= R1);
    const int64_t steps = w + 31;
    for (int64_t k = 0; k < steps; ++k) {
        const int64_t j = k - lane;  // my column offset
        const bool act = (j >= 0 && j < w && r0 <= R1);
        if (lane == 0 && j < w) {
            if (warp == 0) {
                upH = s->top[j + 1].x;
                upF = s->top[j + 1].y;
            } else {
                upH = (int32_t)take(x, &x->bnd[warp - 1][j][0], gen, fail);
                upF = (int32_t)take(x, &x->bnd[warp - 1][j][1], gen, fail);
            }
        }
        int32_t oH = 0, oF = 0;
        if (act) {
            const uint8_t cb = s->cb[j];
            int32_t hd = prevUpH;
            int32_t hu = upH, fu = upF;
            uint32_t word = 0;
#pragma unroll
            for (int i = 0; i < kRW; ++i) {
                if (r0 + i <= R1) {
                    const int32_t eext = El[i] + a.ext, eopen = Hl[i] + a.open;
                    const int32_t fext = fu + a.ext, fopen = hu + a.open;
                    const int32_t e = max(eext, eopen), f = max(fext, fopen);
                    const int32_t dg = hd + (ra[i] == cb ? a.match : a.mismatch);
                    const int32_t hv = max(max(0, e), max(f, dg));
                    word |= ((hv != dg ? BIT_ND : 0u) | (hv != e ? BIT_NE : 0u) | (eext != e ? BIT_NEX : 0u) |
                             (fext != f ? BIT_NFX : 0u))
                            << (4 * i);
                    hd = Hl[i];
                    Hl[i] = hv;
                    El[i] = e;
                    hu = hv;
                    fu = f;
                }
            }
            reinterpret_cast<uint16_t *>(d)[dir_index(t * kRW, (int)j)] = (uint16_t)word;
            oH = hu;
            oF = fu;
            if (publish) {
                x->bnd[warp][j][0] = pack((uint32_t)oH, gen);
                x->bnd[warp][j][1] = pack((uint32_t)oF, gen);
            }
        }
        prevUpH = upH;
        // hand (H, F) of my last row to the lane below for the next step
        const int32_t sH = __shfl_up_sync(0xffffffffu, oH, 1);
        const int32_t sF = __shfl_up_sync(0xffffffffu, oF, 1);
        if (lane > 0) {
            upH = sH;
            upF = sF;
            if (j + 1 == 0) prevUpH = hdiag0;  // my first column: diagonal from the left boundary
        }
    }
}

// The same in packed 16-bit halves, two warps of 256 rows: as in strip16.cuh the low
// halves of a warp are virtual lanes 0..31 (four rows each) and the high halves
// virtual lanes 32..63, and lane 31 turns its slot of the shuffle around.  A
// block's cells lie within 12,000 of its corner (walk16_fits), so offsets from
// base = max(0, corner - 12000) fit, and with base > 0 no H comes down to it, where
// the relu would differ from the recurrence's floor at 0.
// Unrolled by 4: a block walks through its code once, and by 8 a block alone takes
// 35% longer for instruction fetch (600 bp pair's stage 2: 0.176 against 0.129 ms).
// What bounds it: 19 ALU ops a row pair (each direction bit is an exclusive or and
// an unsigned minimum with 1, gathered by a multiply-add) at 64 lanes per SM and cycle,
// and for a block alone the chain of 400 steps.  Stage 2 of the 600 bp pair (one or
// two blocks) 0.26 -> 0.13 ms against the 32-bit recompute, a batch of 24 pairs'
// walker 8.2 -> 2.8 ms.
constexpr int32_t kCornerOffset = 12000;
__device__ __forceinline__ uint32_t dup16(int32_t v) { return (uint32_t)(uint16_t)(int16_t)v * 0x00010001u; }
__device__ __forceinline__ uint32_t pair16(int32_t lo, int32_t hi) {
    return ((uint32_t)(uint16_t)(int16_t)lo) | ((uint32_t)(uint16_t)(int16_t)hi << 16);
}
__device__ __forceinline__ uint32_t prmt(uint32_t lo, uint32_t hi, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return r;
}

// 1 in each half that differs.
__device__ __forceinline__ uint32_t differs(uint32_t a, uint32_t b) { return __vminu2(a ^ b, 0x00010001u); }

struct Lane4 {
    uint32_t H[kRW], E[kRW], ra[kRW];
    uint32_t inH, inF, hd;  // (H, F) of the row above at this column, its H at the previous one
};
struct Scores4 {
    uint32_t open2, ext2, gx2, mt1, mm;
};

// One step: returns the lane's direction word; fl is F of its last rows.  PRED:
// halves whose column is left of the block keep their values (mask).
template <bool PRED>
__device__ __forceinline__ uint32_t step4(Lane4 &L, const Scores4 &c, uint32_t col, uint32_t rv, uint32_t selH,
                                          uint32_t selF, int src, uint32_t mask, uint32_t &fl) {
    uint32_t t[kRW], e[kRW], dg[kRW], word = 0;
    uint32_t hd = L.hd;
#pragma unroll
    for (int i = 0; i < kRW; ++i) {
        const uint32_t s = __viaddmax_s16x2(~(L.ra[i] ^ col), c.mt1, c.mm);
        const uint32_t x = __vadd2(L.E[i], c.ext2);
        e[i] = __viaddmax_s16x2(L.H[i], c.open2, x);
        dg[i] = __vadd2(hd, s);
        t[i] = __vimax_s16x2_relu(dg[i], e[i]);
        word += differs(e[i], x) * (BIT_NEX << (4 * i));
        hd = L.H[i];
    }
    uint32_t y = __vadd2(L.inF, c.ext2);
    uint32_t f = __viaddmax_s16x2(L.inH, c.open2, y);
#pragma unroll
    for (int i = 0; i < kRW; ++i) {
        const uint32_t h = __vmaxs2(t[i], f);
        word += differs(f, y) * (BIT_NFX << (4 * i)) +
                differs(h, dg[i]) * (BIT_ND << (4 * i)) +
                differs(h, e[i]) * (BIT_NE << (4 * i));
        fl = f;
        y = __vadd2(f, c.ext2);
        f = __viaddmax_s16x2(f, c.gx2, __vadd2(t[i], c.open2));
        L.H[i] = PRED ? ((h & mask) | (L.H[i] & ~mask)) : h;
        L.E[i] = PRED ? ((e[i] & mask) | (L.E[i] & ~mask)) : e[i];
    }
    const uint32_t nH = prmt(rv, L.H[kRW - 1], selH), nF = prmt(rv, fl, selF);
    L.hd = L.inH;
    L.inH = __shfl_sync(0xffffffffu, nH, src);
    L.inF = __shfl_sync(0xffffffffu, nF, src);
    return word;
}

// As recompute_wide; kThreads threads.
__device__ void recompute16(const WalkArgs &a, int64_t R0, int64_t R1, int64_t C0, int64_t C1, uint32_t *d, Xchg *x,
                            Stage *s, uint32_t gen) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = (int)(C1 - C0 + 1), h = (int)(R1 - R0 + 1), r_warp = warp * kWarpRows;
    if (r_warp >= h) return;  // this warp has no rows
    const int32_t corner = s->top[0].x, base = max(0, corner - kCornerOffset);
    Scores4 c;
    c.open2 = dup16(a.open);
    c.ext2 = dup16(a.ext);
    c.gx2 = dup16(max(a.open, a.ext));
    c.mt1 = dup16(a.match + 1);
    c.mm = dup16(a.mismatch);
    auto off = [&](int32_t v) { return max(v - base, -16384); };
    if (warp == 0) {
        for (int j = lane; j < w; j += 32) s->top16[j] = pair16(off(s->top[j + 1].x), off(s->top[j + 1].y));
        __syncwarp();
    }
    Lane4 L;
#pragma unroll
    for (int i = 0; i < kRW; ++i) {
        int2 lv[2];
        uint32_t code[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = r_warp + (lane + 32 * q) * kRW + i;  // rows past the end: the last row's boundary, no match
            lv[q] = left_he(a, C0, R0 + min(r, h - 1));
            code[q] = (r < h ? (uint32_t)s->rb[r] : 256u) << 6;
        }
        L.H[i] = pair16(off(lv[0].x), off(lv[1].x));
        L.E[i] = pair16(off(lv[0].y), off(lv[1].y));
        L.ra[i] = code[0] | (code[1] << 16);
    }
    const int src = (lane + 31) & 31;
    const uint32_t selH = lane == 31 ? 0x5410u : 0x7654u, selF = lane == 31 ? 0x5432u : 0x7654u;
    bool fail = false;
    auto above = [&](int j) -> uint32_t {  // (H, F) of the row above the warp at column j
        if (j >= w) j = w - 1;
        return warp == 0 ? s->top16[j] : take(x, &x->bnd[warp - 1][j][0], gen, fail);
    };
    {
        // what the shuffles of the step before column 0 would have brought
        const uint32_t up = __shfl_sync(0xffffffffu, prmt(0u, L.H[kRW - 1], selH), src);
        const int32_t first = warp == 0 ? corner : left_he(a, C0, R0 + r_warp - 1).x;
        const uint32_t v = above(0);
        L.hd = lane == 0 ? prmt((uint32_t)off(first), up, 0x7610u) : up;
        L.inH = lane == 0 ? prmt(v, up, 0x7610u) : up;
        L.inF = v >> 16;
    }
    const bool publish = lane == 31 && r_warp + kWarpRows < h;
    const uint16_t *pc = s->col16 + 64 - lane;
    uint32_t *pd = d + (int64_t)warp * kSteps * 32 + lane;
    unsigned long long(*pub)[2] = x->bnd[warp < kThreads / 32 - 1 ? warp : 0];
    const int steps = w + 63;
    uint32_t col = (uint32_t)pc[0] | ((uint32_t)pc[-32] << 16);
    // chunks of kC steps: one lane per column of the row above; the next step's
    // column codes are loaded ahead.  The last chunk's steps past `steps` write
    // words that no walk reads (kSteps is a multiple of kC).
    for (int k = 0; k < 64; k += kC) {
        const uint32_t ab = above(k + 1 + (lane & (kC - 1)));
        __syncwarp();
#pragma unroll 4
        for (int u = 0; u < kC; ++u) {
            const uint32_t next = (uint32_t)pc[k + u + 1] | ((uint32_t)pc[k + u - 31] << 16);
            const uint32_t rv = __shfl_sync(0xffffffffu, ab, u);
            const uint32_t mask = (k + u >= lane ? 0x0000FFFFu : 0u) | (k + u >= lane + 32 ? 0xFFFF0000u : 0u);
            uint32_t fl;
            pd[(k + u) * 32] = step4<true>(L, c, col, rv, selH, selF, src, mask, fl);
            if (publish && k + u == 63) pub[0][0] = pack(prmt(L.H[kRW - 1], fl, 0x7632u), gen);
            col = next;
        }
    }
    for (int k = 64; k < steps; k += kC) {
        const uint32_t ab = above(k + 1 + (lane & (kC - 1)));
        __syncwarp();
#pragma unroll 4
        for (int u = 0; u < kC; ++u) {
            const uint32_t next = (uint32_t)pc[k + u + 1] | ((uint32_t)pc[k + u - 31] << 16);
            const uint32_t rv = __shfl_sync(0xffffffffu, ab, u);
            uint32_t fl;
            pd[(k + u) * 32] = step4<false>(L, c, col, rv, selH, selF, src, ~0u, fl);
            if (publish && k + u - 63 < w) pub[k + u - 63][0] = pack(prmt(L.H[kRW - 1], fl, 0x7632u), gen);
            col = next;
        }
    }
}

// Either recompute; wide is the same for all blocks of a launch.
template <bool WIDE>
__device__ __forceinline__ void recompute(const WalkArgs &a, int64_t R0, int64_t R1, int64_t C0, int64_t C1, uint32_t *d,
                                          Xchg *x, Stage *s, uint32_t gen) {
    if constexpr (WIDE) recompute_wide(a, R0, R1, C0, C1, d, x, s, gen);
    else recompute16(a, R0, R1, C0, C1, d, x, s, gen);
}

// Warp 0 walks the path through the block that starts at (R0, C0); rb, cb: the
// block's bytes.  Row and column indices fit 32 bits (pairs are limited to
// 2^31 - 64 rows), so the crosspoint tests use 32-bit remainders.
__device__ void walk(const WalkArgs &a, int64_t R0, int64_t C0, const Dir &dir, const uint8_t *rb, const uint8_t *cb,
                     int64_t *S) {
    const int lane = threadIdx.x & 31;
    int64_t r = S[kStR], c = S[kStC];
    int32_t state = (int32_t)S[kStState];
    int64_t nops = S[kStNOps], suffix = S[kStSuffix], nxp = S[kStNXp];
    const int32_t X = a.xp_interval;
    bool done = false, err = false;
    while (!done && !err && r >= R0 && c >= C0) {
        if (state == ST_H) {
            // run of diagonal moves: cells whose H comes from the diagonal, up to the
            // one whose diagonal predecessor has no score left, the start cell
            const int64_t rr = r - lane, cc = c - lane;
            const bool in = rr >= R0 && cc >= C0;
            const uint32_t v = in ? dir.at(rr - R0, cc - C0) : BIT_ND;
            // inclusive prefix over lanes of the substitution scores (the suffix after
            // lane i's cell), from one ballot of the matching cells
            const uint32_t mb = __ballot_sync(0xffffffffu, in && rb[rr - R0] == cb[cc - C0]);
            const uint32_t upto = 0xffffffffu >> (31 - lane);
            const int mle = __popc(mb & upto);
            const int32_t ps = mle * a.match + (lane + 1 - mle) * a.mismatch;
            const uint32_t db = __ballot_sync(0xffffffffu, (v & BIT_ND) == 0);
            const int ndiag = (db == 0xffffffffu) ? 32 : __ffs(~db) - 1;
            const uint32_t sb = __ballot_sync(0xffffffffu, lane < ndiag && (int64_t)a.score == suffix + ps);
            const bool start = sb != 0;
            const int nrun = start ? __ffs(sb) : ndiag;  // cells taken; the start cell is the last
            // crosspoint: moving from (rr, cc) to (rr-1, cc-1) enters row rr-1 from below
            // (not from the start cell)
            const bool xp = lane < nrun - (start ? 1 : 0) && rr - 1 >= 0 && ((int32_t)rr % X) == 0;
            const uint32_t xbal = __ballot_sync(0xffffffffu, xp);
            if (xp) {
                const int64_t slot = nxp + __popc(xbal & ((1u << lane) - 1));
                if (slot < a.xp_cap) {
                    int64_t *d = a.xps + 4 * slot;
                    d[0] = rr - 1;
                    d[1] = cc - 1;
                    d[2] = (int64_t)a.score - (suffix + ps);
                    d[3] = 0;
                }
            }
            if (lane < nrun && nops + lane < a.ops_cap) a.ops[nops + lane] = 'M';
            if (nrun > 0) {
                nops += nrun;
                suffix += __shfl_sync(0xffffffffu, ps, nrun - 1);
                nxp += __popc(xbal);
                r -= nrun;
                c -= nrun;
            }
            if (start) {
                S[kStStartR] = r + 1;
                S[kStStartC] = c + 1;
                done = true;
            } else if (nrun < 32 && r >= R0 && c >= C0) {
                const uint32_t q = dir.at(r - R0, c - C0);
                if (!(q & BIT_ND)) err = true;  // cannot be: the run stopped here
                state = (q & BIT_NE) ? ST_F : ST_E;
            }
        } else if (state == ST_E) {
            // horizontal run: 'I' for every cell until the gap opens
            const int64_t cc = c - lane;
            const bool in = cc >= C0;
            const uint32_t v = in ? dir.at(r - R0, cc - C0) : BIT_NEX;
            const bool ext = !(v & BIT_NEX);
            const uint32_t bal = __ballot_sync(0xffffffffu, ext);
            const uint32_t inb = __ballot_sync(0xffffffffu, in);
            int nrun;                                  // cells consumed
            bool opened;                               // run ended with the gap opening
            const int firstno = (bal == 0xffffffffu) ? 32 : __ffs(~bal) - 1;  // first lane not extending
            if (firstno < 32 && ((inb >> firstno) & 1)) {
                nrun = firstno + 1;
                opened = true;
            } else {
                nrun = min(firstno, __popc(inb));
                opened = false;
            }
            if (lane < nrun && nops + lane < a.ops_cap) a.ops[nops + lane] = 'I';
            nops += nrun;
            suffix += (int64_t)(opened ? nrun - 1 : nrun) * a.ext + (opened ? a.open : 0);
            c -= nrun;
            if (opened) state = ST_H;
        } else {
            // vertical run: 'D' for every cell until the gap opens
            const int64_t rr = r - lane;
            const bool in = rr >= R0;
            const uint32_t v = in ? dir.at(rr - R0, c - C0) : BIT_NFX;
            const bool ext = !(v & BIT_NFX);
            const uint32_t bal = __ballot_sync(0xffffffffu, ext);
            const uint32_t inb = __ballot_sync(0xffffffffu, in);
            const int firstno = (bal == 0xffffffffu) ? 32 : __ffs(~bal) - 1;
            int nrun;
            bool opened;
            if (firstno < 32 && ((inb >> firstno) & 1)) {
                nrun = firstno + 1;
                opened = true;
            } else {
                nrun = min(firstno, __popc(inb));
                opened = false;
            }
            // suffix after lane i's cell: i+1 cells, all ext except an opening cell
            const int64_t cost_i = (int64_t)(lane + 1) * a.ext + ((opened && lane == nrun - 1) ? a.open - a.ext : 0);
            // crosspoint: moving from (rr, c) up to (rr-1, c) enters row rr-1 from below;
            // the cell above is in F if this move extended the gap, else in H
            const bool xp = lane < nrun && rr - 1 >= 0 && ((int32_t)rr % X) == 0;
            const uint32_t xbal = __ballot_sync(0xffffffffu, xp);
            if (xp) {
                const int64_t slot = nxp + __popc(xbal & ((1u << lane) - 1));
                if (slot < a.xp_cap) {
                    int64_t *d = a.xps + 4 * slot;
                    d[0] = rr - 1;
                    d[1] = c;
                    d[2] = (int64_t)a.score - (suffix + cost_i);
                    d[3] = (lane == nrun - 1 && opened) ? 0 : 1;
                }
            }
            if (lane < nrun && nops + lane < a.ops_cap) a.ops[nops + lane] = 'D';
            nops += nrun;
            suffix += (int64_t)(opened ? nrun - 1 : nrun) * a.ext + (opened ? a.open : 0);
            nxp += __popc(xbal);
            r -= nrun;
            if (opened) state = ST_H;
        }
        __syncwarp();
    }
    if (lane == 0) {
        S[kStR] = r;
        S[kStC] = c;
        S[kStState] = state;
        S[kStNOps] = nops;
        S[kStSuffix] = suffix;
        S[kStNXp] = nxp;
        if (done) S[kStDone] = 1;
        if (err) S[kStErr] = 1;
    }
}

// Block after block until the start is reached, the path goes above row r_stop or it
// leaves the region [rr0, .) x [cc0, .).
template <bool WIDE>
__device__ void walk_until(const WalkArgs &a, uint32_t *dir, Xchg *xc, Stage *sg, int64_t *S, int64_t r_stop) {
    int guard = 0;
    for (; guard < (1 << 30); ++guard) {
        const int64_t r = S[kStR], c = S[kStC];
        if (S[kStDone] || S[kStErr] || r < r_stop || r < a.rr0 || c < a.cc0) break;
        const int64_t R0 = a.rr0 + (int64_t)((int32_t)(r - a.rr0) / a.br) * a.br;
        const int64_t C0 = a.cc0 + ((c - a.cc0) / kBC) * kBC;
        stage_block(a, R0, r, C0, c, sg);
        __syncthreads();
        recompute<WIDE>(a, R0, r, C0, c, dir, xc, sg, xc->gen + (uint32_t)guard + 1u);
        __syncthreads();
        if (xc->err) {
            if (threadIdx.x == 0) S[kStErr] = 1;
            __syncthreads();
            break;
        }
        if (threadIdx.x < 32) walk(a, R0, C0, Dir{dir}, sg->rb, sg->cb, S);
        __syncthreads();
    }
    __syncthreads();
    if (threadIdx.x == 0) xc->gen += (uint32_t)guard + 1u;  // generations used here
    __syncthreads();
}

// Precomputes the directions of whole blocks (R0, C0) = blk[2b], blk[2b + 1]
// of a region into gdir + b * kBlockWords (one CTA per block at a time).  A block
// depends only on the stored boundaries, not on the path, so any set of blocks
// can run at once.
template <bool WIDE>
__global__ void __launch_bounds__(WIDE ? kThreadsWide : kThreads) precompute_kernel(WalkArgs a, const int64_t *blk,
                                                                                   int64_t nblk, uint32_t *gdir,
                                                                                   int32_t *err) {
    __shared__ Xchg xc;
    __shared__ Stage sg;
    xchg_init(&xc);
    uint32_t gen = 0;
    for (int64_t b = blockIdx.x; b < nblk; b += gridDim.x) {
        const int64_t R0 = blk[2 * b], C0 = blk[2 * b + 1];
        const int64_t R1 = min(R0 + a.br - 1, a.rr1 - 1), C1 = min(C0 + kBC - 1, a.cc1 - 1);
        __syncthreads();
        stage_block(a, R0, R1, C0, C1, &sg);
        __syncthreads();
        recompute<WIDE>(a, R0, R1, C0, C1, gdir + b * kBlockWords, &xc, &sg, ++gen);
    }
    __syncthreads();
    if (threadIdx.x == 0 && xc.err) atomicExch(err, 1);
}

// The same for blocks of several regions (level-1 cells): reg[b] is block b's.
template <bool WIDE>
__global__ void __launch_bounds__(WIDE ? kThreadsWide : kThreads)
    precompute_cells_kernel(const WalkArgs *regs, const int64_t *blk, const int32_t *reg, int64_t nblk, uint32_t *gdir,
                            int32_t *err) {
    __shared__ Xchg xc;
    __shared__ Stage sg;
    __shared__ WalkArgs a;
    xchg_init(&xc);
    uint32_t gen = 0;
    for (int64_t b = blockIdx.x; b < nblk; b += gridDim.x) {
        __syncthreads();
        if (threadIdx.x == 0) a = regs[reg[b]];
        __syncthreads();
        const int64_t R0 = blk[2 * b], C0 = blk[2 * b + 1];
        const int64_t R1 = min(R0 + a.br - 1, a.rr1 - 1), C1 = min(C0 + kBC - 1, a.cc1 - 1);
        stage_block(a, R0, R1, C0, C1, &sg);
        __syncthreads();
        recompute<WIDE>(a, R0, R1, C0, C1, gdir + b * kBlockWords, &xc, &sg, ++gen);
    }
    __syncthreads();
    if (threadIdx.x == 0 && xc.err) atomicExch(err, 1);
}

// One warp walks the path through precomputed blocks: block (bi, bj) of the
// region (relative to rr0, cc0) is slot map[(bi - bi0) * mw + (bj - bj0)] of
// gdir, or absent (-1).  Stops where the path enters an absent block, at the
// start cell or on an error; the state is read from and written back to a.st.
// Waits (bounded) for phase `parity` of the mbarrier at shared address bar.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > kXchgWaitCycles) return false;
    }
}

// The aligned word at p of the sequence bytes [lo, hi); bytes outside are not read.
__device__ __forceinline__ uint32_t seq_word(const uint8_t *lo, const uint8_t *hi, const uint32_t *p) {
    const uint8_t *b = reinterpret_cast<const uint8_t *>(p);
    if (b >= lo && b + 4 <= hi) return *p;
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (b + k >= lo && b + k < hi) v |= (uint32_t)b[k] << (8 * k);
    return v;
}

// The walk of each block reads the block's direction words from shared memory:
// on entering a block the warp copies the part the path can still reach (the
// 256-row chunks at or above the current row, the steps up to the current
// column + 63) from gdir with one bulk asynchronous copy (cp.async.bulk, the
// TMA engine) per chunk, completing on an mbarrier; every step of the walk is
// then a shared-memory read instead of a dependent L2 round trip.  The block's
// sequence bytes, for the path's scores, are fetched as aligned words while the
// copy is on its way.
__global__ void __launch_bounds__(32) corridor_walk_kernel(WalkArgs a, const uint32_t *gdir, const int32_t *map,
                                                           int64_t bi0, int64_t bj0, int64_t mh, int64_t mw,
                                                           const int32_t *err) {
    extern __shared__ __align__(16) uint32_t dtile[];  // kBlockWords words
    __shared__ uint32_t seq_r[kBR / 4 + 2], seq_c[kBC / 4 + 2];
    __shared__ int64_t S[kStN];
    __shared__ __align__(8) uint64_t bar_mem;
    const int lane = threadIdx.x;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&bar_mem);
    if (lane < kStN) S[lane] = a.st[lane];
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (*err) {
        if (lane == 0) S[kStErr] = 1;
        __syncwarp();
    }
    uint32_t phase = 0;
    bool in_flight = false;
    for (;;) {
        const int64_t r = S[kStR], c = S[kStC];
        if (S[kStDone] || S[kStErr] || r < a.rr0 || c < a.cc0) break;
        // region offsets fit 32 bits: 32-bit division
        const int64_t bi = (int32_t)(r - a.rr0) / a.br, bj = (c - a.cc0) / kBC;
        if (bi < bi0 || bi >= bi0 + mh || bj < bj0 || bj >= bj0 + mw) break;
        const int32_t slot = map[(bi - bi0) * mw + (bj - bj0)];
        if (slot < 0) break;
        const int64_t R0 = a.rr0 + bi * a.br, C0 = a.cc0 + bj * kBC;
        const int wmax = (int)((r - R0) / kWarpRows);
        const int kn = (int)(c - C0) + 64;
        const uint32_t chunk = (uint32_t)kn * 32u * 4u;
        __syncwarp();  // the previous block's reads of dtile are done
        if (lane == 0) {
            const uint32_t *src = gdir + (int64_t)slot * kBlockWords;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                         "r"((uint32_t)(wmax + 1) * chunk)
                         : "memory");
            for (int w = 0; w <= wmax; ++w)
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        (uint32_t)__cvta_generic_to_shared(dtile + (int64_t)w * kSteps * 32)),
                    "l"(src + (int64_t)w * kSteps * 32), "r"(chunk), "r"(bar)
                    : "memory");
        }
        in_flight = true;
        // bytes R0..r and C0..c, as the aligned words that hold them
        const uintptr_t pr = reinterpret_cast<uintptr_t>(a.rows + R0), pc = reinterpret_cast<uintptr_t>(a.cols + C0);
        const int nr = (int)((pr & 3) + (r - R0)) / 4 + 1, nc = (int)((pc & 3) + (c - C0)) / 4 + 1;
        {
            uint32_t v[kBR / 128 + 1 + kBC / 128 + 1];
            constexpr int kNR = kBR / 128 + 1, kNC = kBC / 128 + 1;
#pragma unroll
            for (int q = 0; q < kNR; ++q)
                if (lane + 32 * q < nr)
                    v[q] = seq_word(a.rows, a.rows + a.m, reinterpret_cast<const uint32_t *>(pr & ~(uintptr_t)3) + lane + 32 * q);
#pragma unroll
            for (int q = 0; q < kNC; ++q)
                if (lane + 32 * q < nc)
                    v[kNR + q] = seq_word(a.cols, a.cols + a.n, reinterpret_cast<const uint32_t *>(pc & ~(uintptr_t)3) + lane + 32 * q);
#pragma unroll
            for (int q = 0; q < kNR; ++q)
                if (lane + 32 * q < nr) seq_r[lane + 32 * q] = v[q];
#pragma unroll
            for (int q = 0; q < kNC; ++q)
                if (lane + 32 * q < nc) seq_c[lane + 32 * q] = v[kNR + q];
        }
        const bool ok = __all_sync(0xffffffffu, bar_wait(bar, phase & 1));
        if (!ok) {
            if (lane == 0) S[kStErr] = 1;
            __syncwarp();
            break;
        }
        in_flight = false;
        ++phase;
        __syncwarp();
        walk(a, R0, C0, Dir{dtile}, reinterpret_cast<const uint8_t *>(seq_r) + (pr & 3),
             reinterpret_cast<const uint8_t *>(seq_c) + (pc & 3), S);
        __syncwarp();
    }
    // A copy still in flight after its wait ran out writes this CTA's shared
    // memory, so the warp waits for it once more before the CTA exits.  It reads
    // at most kBlockWords words of this GPU's own memory and lands in
    // microseconds; every wait of the library is bounded (here about 1 s), and a
    // copy that has not landed after two bounds means the device is failing: the
    // error stays set for the host.
    if (in_flight && !__all_sync(0xffffffffu, bar_wait(bar, phase & 1)) && lane == 0) S[kStErr] = 1;
    __syncwarp();
    if (lane < kStN) a.st[lane] = S[lane];
}

// ------------------------------------------------------------------ segments
//
// A walk is serial from the end cell, but where the path crosses a special row can
// be guessed: along an alignment the row's highest H near the expected diagonal is
// the path's, or a few cells off, and a traceback from there runs into the path
// within a few rows.  So the rows of a pair are cut at its special rows into
// segments that are walked at the same time, each from its guess up to the next
// special row; a second round walks every segment again whose entry is not where
// the segment below left it.  Nothing is taken on trust: a segment counts only
// when its entry cell and state are the exit of the segment below, starting at the
// true end cell; the others are walked serially.  Stage 2 against one warp walking
// the whole path: 1 Mbp pair 26.6 -> 2.6 ms, 172 kbp pair 4.3 -> 0.7 ms, a batch of
// 24 pairs 2.7 -> 0.5 ms.

struct SegRec {
    int64_t er, ec, xr, xc, sr, sc;  // entry cell, exit cell, start cell (done)
    int32_t est, xst;                // walk state at entry and exit
    int32_t val, xval;               // H (or F) of the entry, and the path's prefix score at the exit
    int32_t nops, nxp;
    int32_t valid, done;
};
constexpr int kSegOps = 4096;  // operations and crosspoints a segment may hold
constexpr int kSegXps = 160;
// A pair alone: below this many segments one corridor of precomputed blocks is as fast.
constexpr int kSegPairMin = 8;
constexpr int kSegChain = 32;  // records a batched pair's CTA looks at together
// Segments of one launch (9.4 KB of records and outputs each): of a batch, and of a
// pair walked alone, which takes its segments in windows from its current row up.
constexpr int64_t kSegMax = 65536, kSegWindow = 4096;
constexpr int kSegMin = 3;     // segments a pair must have to be walked in segments

struct SegArgs {
    const WalkArgs *args;       // per pair; st holds the end cell (or the cell reached so far)
    const int2 *items;          // (pair, segment)
    int64_t nitems;
    const int32_t *base;        // per pair: its first segment's index; -1: no segments
    SegRec *rec[2];             // per segment: read and written by alternate rounds
    char *ops;                  // per segment: kSegOps bytes
    int64_t *xps;               // per segment: kSegXps crosspoints
    uint32_t *gdir;             // kBlockWords words per CTA
};

// Column of the highest H of special row q (its row is (q + 1) * br - 1) near the
// diagonal through (r, c); -1 when there is none.  All threads; sh: one slot per warp.
__device__ int64_t guess_column(const WalkArgs &a, int64_t q, int64_t r, int64_t c, unsigned long long *sh) {
    const int64_t er = (q + 1) * a.br - 1, d = r - er, mid = c - d, w = 512 + d / 16;
    const int64_t lo = max((int64_t)0, mid - w), hi = min(a.cc1 - 1, mid + w);
    const int2 *row = a.srows + q * a.cc1;
    unsigned long long best = 0;
    constexpr int kN = 4;
    for (int64_t j0 = lo + threadIdx.x; j0 <= hi; j0 += kN * blockDim.x) {
        int32_t h[kN];
#pragma unroll
        for (int k = 0; k < kN; ++k) h[k] = j0 + k * blockDim.x <= hi ? row[j0 + k * blockDim.x].x : 0;
#pragma unroll
        for (int k = 0; k < kN; ++k) {
            const unsigned long long v = ((unsigned long long)(uint32_t)h[k] << 32) | (uint32_t)(j0 + k * blockDim.x);
            best = max(best, v);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, off));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = best;
    __syncthreads();
    for (int k = 0; k < (int)blockDim.x / 32; ++k) best = max(best, sh[k]);
    __syncthreads();
    return (best >> 32) ? (int64_t)(uint32_t)best : -1;
}

// One round over the segments: GUESS from the special rows, or every segment from
// the exit of the one below it in `in`.
template <bool WIDE, bool GUESS>
__device__ __forceinline__ void walk_segments(const SegArgs &g, const SegRec *in, SegRec *out) {
    __shared__ Xchg xc;
    __shared__ Stage sg;
    __shared__ int64_t S[kStN];
    __shared__ WalkArgs sa;
    __shared__ SegRec rec;
    __shared__ unsigned long long sh[kThreadsWide / 32];
    xchg_init(&xc);
    uint32_t *dir = g.gdir + (int64_t)blockIdx.x * kBlockWords;
    for (int64_t it = blockIdx.x; it < g.nitems; it += gridDim.x) {
        const int2 item = g.items[it];
        const int64_t q = item.y, slot = g.base[item.x] + q;
        __syncthreads();
        if (threadIdx.x == 0) {
            sa = g.args[item.x];
            xc.err = 0;
        }
        __syncthreads();
        const int64_t *st = sa.st;
        const int64_t r = st[kStR], c = st[kStC], bottom = r < 0 ? -1 : r / sa.br;
        if (st[kStDone] || q > bottom) continue;
        SegRec e{};
        if (q == bottom) {
            e.er = r;
            e.ec = c;
            e.est = (int32_t)st[kStState];
            e.val = (int32_t)(sa.score - st[kStSuffix]);
            e.valid = 1;
        } else if (GUESS) {
            e.er = (q + 1) * sa.br - 1;
            e.ec = guess_column(sa, q, r, c, sh);
            e.est = ST_H;
            e.valid = e.ec >= 0;
        } else {
            const SegRec lower = in[slot + 1];
            e.er = lower.xr;
            e.ec = lower.xc;
            e.est = lower.xst;
            e.valid = lower.valid && !lower.done && lower.xc >= 0 && lower.xr == (q + 1) * sa.br - 1;
        }
        if (!GUESS) {
            const SegRec old = in[slot];
            if (!e.valid || (old.valid && old.er == e.er && old.ec == e.ec && old.est == e.est)) {
                // (a segment nothing leads into keeps its record: its operations still stand)
                if (threadIdx.x == 0) out[slot] = old;
                continue;
            }
        }
        if (!e.valid) {
            if (threadIdx.x == 0) out[slot] = e;
            continue;
        }
        if (q != bottom) {
            const int2 hf = sa.srows[q * sa.cc1 + e.ec];
            e.val = e.est == ST_F ? hf.y : hf.x;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            rec = e;
            sa.score = e.val;
            sa.ops = g.ops + slot * kSegOps;
            sa.ops_cap = kSegOps;
            sa.xps = g.xps + slot * kSegXps * 4;
            sa.xp_cap = kSegXps;
            for (int k = 0; k < kStN; ++k) S[k] = 0;
            S[kStR] = e.er;
            S[kStC] = e.ec;
            S[kStState] = e.est;
        }
        __syncthreads();
        walk_until<WIDE>(sa, dir, &xc, &sg, S, q * sa.br);
        if (threadIdx.x == 0) {
            rec.xr = S[kStR];
            rec.xc = S[kStC];
            rec.xst = (int32_t)S[kStState];
            rec.sr = S[kStStartR];
            rec.sc = S[kStStartC];
            rec.xval = (int32_t)(rec.val - S[kStSuffix]);
            rec.nops = (int32_t)min(S[kStNOps], (int64_t)INT_MAX);
            rec.nxp = (int32_t)min(S[kStNXp], (int64_t)INT_MAX);
            rec.done = S[kStDone] != 0;
            rec.valid = !S[kStErr] && rec.nops <= kSegOps && rec.nxp <= kSegXps;
            out[slot] = rec;
        }
        __syncthreads();
    }
}

template <bool WIDE, bool GUESS>
__global__ void __launch_bounds__(WIDE ? kThreadsWide : kThreads) seg_kernel(SegArgs g, int in) {
    walk_segments<WIDE, GUESS>(g, g.rec[in], g.rec[in ^ 1]);
}

// Copies accepted segments' operations and crosspoints to their places: segment
// (first - b) of block b goes to ops + off[2b], xps + 4 off[2b + 1].
__global__ void seg_copy_kernel(const SegRec *rec, const char *sops, const int64_t *sxps, int64_t first, const int64_t *off,
                                char *ops, int64_t *xps) {
    const int64_t slot = first - blockIdx.x;
    const int nops = rec[slot].nops, nx = 4 * rec[slot].nxp;
    char *po = ops + off[2 * blockIdx.x];
    int64_t *px = xps + 4 * off[2 * blockIdx.x + 1];
    for (int i = threadIdx.x; i < nops; i += blockDim.x) po[i] = sops[slot * kSegOps + i];
    for (int i = threadIdx.x; i < nx; i += blockDim.x) px[i] = sxps[slot * kSegXps * 4 + i];
}

// A walked pair's results in their final form: operations start -> end at
// ops + off.ops, crosspoints [start, top -> bottom, end] at xps + off.xps.
struct PackOff {
    int64_t ops, xps, end_r, end_c;
};
__global__ void pack_results_kernel(const WalkArgs *args, const PackOff *offs, char *ops, swb_xpoint *xps) {
    const WalkArgs &a = args[blockIdx.x];
    const PackOff o = offs[blockIdx.x];
    const int64_t nops = a.st[kStNOps], nxp = a.st[kStNXp];
    for (int64_t i = threadIdx.x; i < nops; i += blockDim.x) ops[o.ops + i] = a.ops[nops - 1 - i];
    swb_xpoint *x = xps + o.xps;
    for (int64_t i = threadIdx.x; i < nxp; i += blockDim.x) {
        const int64_t *d = a.xps + 4 * (nxp - 1 - i);
        x[1 + i] = swb_xpoint{(int32_t)d[3], (int32_t)d[2], d[0], d[1]};
    }
    if (threadIdx.x == 0) {
        x[0] = swb_xpoint{0, 0, a.st[kStStartR], a.st[kStStartC]};
        x[1 + nxp] = swb_xpoint{0, a.score, o.end_r, o.end_c};
    }
}

// Batched pairs: CTA b walks pairs b, b + gridDim.x, ... (each pair's whole matrix is
// its region), recomputing the blocks on its path on demand into its own region of
// gdir (kBlockWords words per CTA).  With segments (g), the ones that continue the
// path are taken over and only the others walked.
template <bool WIDE>
__device__ __forceinline__ void walk_pairs(const WalkArgs *args, int64_t n, uint32_t *gdir, const SegArgs *g) {
    __shared__ Xchg xc;
    __shared__ Stage sg;
    __shared__ int64_t S[kStN];
    __shared__ WalkArgs sa;
    __shared__ SegRec chain[kSegChain];
    __shared__ int64_t at_ops[kSegChain], at_xps[kSegChain];
    __shared__ int taken;
    xchg_init(&xc);
    uint32_t *dir = gdir + (int64_t)blockIdx.x * kBlockWords;
    for (int64_t p = blockIdx.x; p < n; p += gridDim.x) {
        __syncthreads();
        if (threadIdx.x == 0) {
            sa = args[p];
            xc.err = 0;
        }
        __syncthreads();
        if (threadIdx.x < kStN) S[threadIdx.x] = sa.st[threadIdx.x];
        __syncthreads();
        const int64_t base = g ? g->base[p] : -1;
        if (base < 0) walk_until<WIDE>(sa, dir, &xc, &sg, S, 0);
        while (base >= 0 && !S[kStDone] && !S[kStErr] && S[kStR] >= 0 && S[kStC] >= 0) {
            // the next segments' records, the ones of them that continue the path, and
            // their outputs, a warp a segment
            const int64_t q = S[kStR] / sa.br;
            const int k = (int)min((int64_t)kSegChain, q + 1);
            for (int i = threadIdx.x; i < k * (int)(sizeof(SegRec) / 8); i += blockDim.x)
                reinterpret_cast<int64_t *>(chain)[i] = reinterpret_cast<const int64_t *>(g->rec[0] + base + q + 1 - k)[i];
            __syncthreads();
            if (threadIdx.x == 0) {
                int took = 0;
                while (took < k && !S[kStDone]) {
                    const SegRec &e = chain[k - 1 - took];
                    if (!(e.valid && e.er == S[kStR] && e.ec == S[kStC] && e.est == S[kStState] &&
                          e.val == sa.score - S[kStSuffix]))
                        break;
                    at_ops[took] = S[kStNOps];
                    at_xps[took] = S[kStNXp];
                    S[kStR] = e.xr;
                    S[kStC] = e.xc;
                    S[kStState] = e.xst;
                    S[kStNOps] += e.nops;
                    S[kStNXp] += e.nxp;
                    S[kStSuffix] += e.val - e.xval;
                    if (e.done) {
                        S[kStDone] = 1;
                        S[kStStartR] = e.sr;
                        S[kStStartC] = e.sc;
                    }
                    ++took;
                }
                taken = took;
            }
            __syncthreads();
            const int lane = threadIdx.x & 31;
            for (int t = threadIdx.x >> 5; t < taken; t += blockDim.x / 32) {
                const SegRec &e = chain[k - 1 - t];
                const char *so = g->ops + (base + q - t) * kSegOps;
                const int64_t *sx = g->xps + (base + q - t) * kSegXps * 4;
                const int64_t nops = at_ops[t], nxp = at_xps[t];
                for (int i = lane; i < e.nops; i += 32)
                    if (nops + i < sa.ops_cap) sa.ops[nops + i] = so[i];
                for (int i = lane; i < 4 * e.nxp; i += 32)
                    if (nxp + i / 4 < sa.xp_cap) sa.xps[4 * nxp + i] = sx[i];
            }
            const bool walk_on = taken == 0;
            __syncthreads();
            if (walk_on) walk_until<WIDE>(sa, dir, &xc, &sg, S, q * sa.br);
        }
        if (threadIdx.x < kStN) sa.st[threadIdx.x] = S[threadIdx.x];
        __syncthreads();
    }
}

template <bool WIDE>
__global__ void __launch_bounds__(WIDE ? kThreadsWide : kThreads) walk_batch_kernel(const WalkArgs *args, int64_t n,
                                                                                   uint32_t *gdir, SegArgs g) {
    walk_pairs<WIDE>(args, n, gdir, g.nitems > 0 ? &g : nullptr);
}

// Graphed batches: every pair's walk starts at the best cell the scoring kernel
// merged into pbest (a pair without a positive score is marked done at once).  After a
// scoring kernel that gave up (an error code in the control words) neither the best
// cells nor the stores are all written: every pair is marked done, so that nothing
// walks, and the host reads the code.
__global__ void walk_graph_init_kernel(const GraphHdr *h) {
    const int64_t np = h->npairs;
    WalkArgs *args = (WalkArgs *)h->walk_args;
    int64_t *st = h->walk_states;
    const int32_t open = h->ba.open;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np; p += stride) {
        const BestRec b = h->pbest[p];
        const int32_t score = b.valid && h->out[1] == 0 ? b.ho - open : 0;
        args[p].score = score;
        int64_t *S = st + p * kStN;
#pragma unroll
        for (int k = 0; k < kStN; ++k) S[k] = 0;
        S[kStR] = b.row;
        S[kStC] = b.col;
        if (score <= 0) S[kStDone] = 1;
    }
}

__device__ __forceinline__ SegArgs seg_args(const GraphHdr *h) {
    SegArgs g{};
    g.args = (const WalkArgs *)h->walk_args;
    g.items = h->seg_items;
    g.nitems = h->seg_nitems;
    g.base = h->seg_base;
    g.rec[0] = (SegRec *)h->seg_rec;
    g.rec[1] = (SegRec *)h->seg_rec + h->seg_nitems;
    g.ops = (char *)((SegRec *)h->seg_rec + 2 * h->seg_nitems);
    g.xps = (int64_t *)(g.ops + h->seg_nitems * kSegOps);
    g.gdir = h->walk_dir;
    return g;
}

template <bool WIDE>
__global__ void __launch_bounds__(WIDE ? kThreadsWide : kThreads) walk_graph_kernel(const GraphHdr *h) {
    const SegArgs g = seg_args(h);
    walk_pairs<WIDE>((const WalkArgs *)h->walk_args, h->npairs, h->walk_dir, g.nitems > 0 ? &g : nullptr);
}

template <bool WIDE, bool GUESS>
__global__ void __launch_bounds__(WIDE ? kThreadsWide : kThreads) seg_graph_kernel(const GraphHdr *h, int in) {
    const SegArgs g = seg_args(h);
    walk_segments<WIDE, GUESS>(g, g.rec[in], g.rec[in ^ 1]);
}

}  // namespace

cudaError_t walker_configure() {
    const int c = cudaSharedmemCarveoutMaxShared;
    const auto A = cudaFuncAttributePreferredSharedMemoryCarveout;
    cudaError_t e = cudaSuccess;
    for (cudaError_t x : {cudaFuncSetAttribute((const void *)precompute_kernel<false>, A, c),
                          cudaFuncSetAttribute((const void *)precompute_kernel<true>, A, c),
                          cudaFuncSetAttribute((const void *)precompute_cells_kernel<false>, A, c),
                          cudaFuncSetAttribute((const void *)precompute_cells_kernel<true>, A, c),
                          cudaFuncSetAttribute((const void *)corridor_walk_kernel, A, c),
                          cudaFuncSetAttribute((const void *)corridor_walk_kernel,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirTileBytes),
                          cudaFuncSetAttribute((const void *)walk_batch_kernel<false>, A, c),
                          cudaFuncSetAttribute((const void *)walk_batch_kernel<true>, A, c),
                          cudaFuncSetAttribute((const void *)walk_graph_kernel<false>, A, c),
                          cudaFuncSetAttribute((const void *)walk_graph_kernel<true>, A, c),
                          cudaFuncSetAttribute((const void *)walk_graph_init_kernel, A, c),
                          cudaFuncSetAttribute((const void *)seg_kernel<false, false>, A, c),
                          cudaFuncSetAttribute((const void *)seg_kernel<false, true>, A, c),
                          cudaFuncSetAttribute((const void *)seg_kernel<true, false>, A, c),
                          cudaFuncSetAttribute((const void *)seg_kernel<true, true>, A, c),
                          cudaFuncSetAttribute((const void *)seg_graph_kernel<false, false>, A, c),
                          cudaFuncSetAttribute((const void *)seg_graph_kernel<false, true>, A, c),
                          cudaFuncSetAttribute((const void *)seg_graph_kernel<true, false>, A, c),
                          cudaFuncSetAttribute((const void *)seg_graph_kernel<true, true>, A, c),
                          cudaFuncSetAttribute((const void *)seg_copy_kernel, A, c),
                          cudaFuncSetAttribute((const void *)pack_results_kernel, A, c)})
        if (x != cudaSuccess) e = x;
    return e;
}

bool spill_placement(uint64_t hbm, uint64_t spill, uint64_t rows_bytes, uint64_t cols_bytes, bool *rows_host,
                     bool *cols_host) {
    *rows_host = *cols_host = false;
    if (rows_bytes + cols_bytes <= hbm) return true;
    if (rows_bytes <= spill && cols_bytes <= hbm) return *rows_host = true;
    if (cols_bytes <= spill && rows_bytes <= hbm) return *cols_host = true;
    if (rows_bytes + cols_bytes <= spill) return *rows_host = *cols_host = true;
    return false;
}

Plan plan_for(const swb_options &opts, int64_t m, int64_t n, int64_t br) {
    Plan p;
    if (br <= 0 || br > kBR || br % 32 != 0) br = kBR;
    const double budget = (double)(opts.hbm_budget_bytes ? opts.hbm_budget_bytes : (64ULL << 30));
    const uint64_t rows_bytes = 8ULL * (uint64_t)(m / br) * (uint64_t)n;
    const uint64_t cols_bytes = 8ULL * (uint64_t)(n / kBC) * (uint64_t)m;
    bool rh = false, ch = false;
    if (spill_placement((uint64_t)budget, opts.host_spill_bytes, rows_bytes, cols_bytes, &rh, &ch)) {
        p.level1 = false;
        p.kr = br;
        p.kc = kBC;
        p.br = br;
        return p;
    }
    p.br = kBR;
    // level 1: multiples of the block grid sized to the budget (half rows, half
    // columns).  The row spacing starts at 3584 = 7 x 512 = 8 x 448 rows, so stage
    // 1 may run 448-row strips as well as 512- or 256-row ones, while each level-1
    // cell is recomputed with 512-row blocks.
    p.level1 = true;
    int64_t kr = 7 * kBR, kc = kBC;
    while (8.0 * (double)(m / kr) * (double)n > budget / 2) kr *= 2;
    while (8.0 * (double)(n / kc) * (double)m > budget / 2) kc *= 2;
    p.kr = kr;
    p.kc = kc;
    return p;
}

// Block rows of a region's grid: in.br, or the full block height when unset.
static int64_t block_rows_of(const WalkInputs &in) { return in.br > 0 && in.br <= kBR ? in.br : kBR; }

// Whether a block's cells stay within kCornerOffset of its corner (the spread bound
// of strip16.cuh over the block's rows and columns) and the scores fit the packed
// recompute.
bool walk16_fits(const swb_scoring &sc) {
    const int64_t e = std::min(-(int64_t)sc.gap_open, -(int64_t)sc.gap_extend);
    const int64_t slope = sc.match + e, open = -(int64_t)sc.gap_open;
    return (kBR + kBC + 2) * slope + 3 * open - sc.gap_extend <= kCornerOffset - 256 && sc.match - sc.mismatch <= 64 &&
           sc.gap_extend >= -1000 && open <= 1000 && sc.mismatch >= -1000;
}

static WalkArgs to_args(const WalkInputs &in) {
    WalkArgs a{};
    a.rows = in.rows;
    a.cols = in.cols;
    a.m = in.m;
    a.n = in.n;
    a.match = in.sc.match;
    a.mismatch = in.sc.mismatch;
    a.open = in.sc.gap_open;
    a.ext = in.sc.gap_extend;
    a.score = in.score;
    a.srows = in.srows;
    a.scols = in.scols;
    a.rr0 = in.rr0;
    a.cc0 = in.cc0;
    a.rr1 = in.rr1;
    a.cc1 = in.cc1;
    a.rtop = in.rtop;
    a.rleft = in.rleft;
    a.xp_interval = in.xp_interval;
    a.ops = in.ops;
    a.ops_cap = in.ops_cap;
    a.xps = in.xps;
    a.xp_cap = in.xp_cap;
    a.st = in.dstate;
    a.br = (int32_t)block_rows_of(in);
    a.wide = walk16_fits(in.sc) ? 0 : 1;
    return a;
}

// Blocks the path is expected to cross next: the staircase of blocks along the
// diagonal from the current cell toward the region's origin (a local alignment
// of related sequences runs close to a diagonal), with the block above and the
// block to the left of each as margin, in walk order, at most `cap` of them.
static void predict_corridor(const WalkInputs &in, int64_t r, int64_t c, int64_t cap, std::vector<int64_t> &blk,
                             int64_t &bi0, int64_t &bj0, int64_t &mh, int64_t &mw, std::vector<int32_t> &map) {
    const int64_t BR = block_rows_of(in);
    std::vector<std::pair<int64_t, int64_t>> list;
    auto add = [&](int64_t bi, int64_t bj) {
        if (bi < 0 || bj < 0 || (int64_t)list.size() >= cap) return;
        for (size_t q = list.size() >= 8 ? list.size() - 8 : 0; q < list.size(); ++q)
            if (list[q].first == bi && list[q].second == bj) return;
        list.emplace_back(bi, bj);
    };
    int64_t bi = (r - in.rr0) / BR, bj = (c - in.cc0) / kBC;
    add(bi, bj);
    add(bi - 1, bj);
    add(bi, bj - 1);
    while ((int64_t)list.size() < cap) {
        const int64_t R0 = in.rr0 + bi * BR, C0 = in.cc0 + bj * kBC;
        const int64_t d = std::min(r - R0 + 1, c - C0 + 1);
        r -= d;
        c -= d;
        if (r < in.rr0 || c < in.cc0) break;
        bi = (r - in.rr0) / BR;
        bj = (c - in.cc0) / kBC;
        add(bi, bj);
        add(bi - 1, bj);
        add(bi, bj - 1);
    }
    int64_t bmin = INT64_MAX, bmax = -1, cmin = INT64_MAX, cmax = -1;
    for (auto &p : list) {
        bmin = std::min(bmin, p.first);
        bmax = std::max(bmax, p.first);
        cmin = std::min(cmin, p.second);
        cmax = std::max(cmax, p.second);
    }
    bi0 = bmin;
    bj0 = cmin;
    mh = bmax - bmin + 1;
    mw = cmax - cmin + 1;
    map.assign((size_t)(mh * mw), -1);
    blk.resize(2 * list.size());
    for (size_t q = 0; q < list.size(); ++q) {
        int32_t &slot = map[(size_t)((list[q].first - bi0) * mw + (list[q].second - bj0))];
        if (slot < 0) slot = (int32_t)q;
        blk[2 * q] = in.rr0 + list[q].first * BR;
        blk[2 * q + 1] = in.cc0 + list[q].second * kBC;
    }
}

// A guess round into the second records, a propagating round into the first.
static void launch_segments(const SegArgs &g, bool wide, int64_t grid, cudaStream_t st) {
    if (wide) {
        seg_kernel<true, true><<<(unsigned)grid, kThreadsWide, 0, st>>>(g, 0);
        seg_kernel<true, false><<<(unsigned)grid, kThreadsWide, 0, st>>>(g, 1);
    } else {
        seg_kernel<false, true><<<(unsigned)grid, kThreads, 0, st>>>(g, 0);
        seg_kernel<false, false><<<(unsigned)grid, kThreads, 0, st>>>(g, 1);
    }
}

// Segments of a pair from host_state's cell up, a window of them: takes over the ones
// that continue the path and returns their number in *taken, or -1 when there are too
// few of them or no memory for them (the pair is walked without).  in.dstate holds
// host_state; gdir: blocks of walk_graph_ctas(sms) CTAs.
static int walk_pair_segments(cudaStream_t st, int sms, const WalkInputs &in, const WalkArgs &a, int64_t *host_state,
                              uint32_t *gdir, const Scratch &scr, std::string &err, int32_t *launches, int64_t *taken) {
    cudaError_t e;
    *taken = -1;
    // up to the rows for which guess_column still looks inside the matrix
    const int64_t top = host_state[kStR] / a.br, reach = (host_state[kStC] + 512) * 16 / 15 / a.br + 2;
    const int64_t nseg = std::min({top + 1, reach, kSegWindow, (int64_t)(in.seg_bytes / seg_scratch_bytes(1))});
    if (nseg < kSegPairMin) return SWB_OK;
    const int64_t q0 = top + 1 - nseg, grid = std::min<int64_t>(nseg, walk_graph_ctas(sms));
    SegRec *rec = (SegRec *)scr.ensure(scr.owner, kScrSegRec, seg_scratch_bytes(nseg));
    char *d_items = (char *)scr.ensure(scr.owner, kScrSegItems, sizeof(WalkArgs) + 16 + sizeof(int2) * (size_t)nseg);
    int64_t *d_off = (int64_t *)scr.ensure(scr.owner, kScrSegOff, sizeof(int64_t) * 2 * (size_t)nseg);
    if (!rec || !d_items || !d_off) {
        cudaGetLastError();
        return SWB_OK;
    }
    *taken = 0;
    std::vector<char> up(sizeof(WalkArgs) + 16 + sizeof(int2) * (size_t)nseg, 0);
    std::memcpy(up.data(), &a, sizeof a);
    const int32_t base = (int32_t)-q0;  // segment q's record is base + q
    std::memcpy(up.data() + sizeof(WalkArgs), &base, sizeof base);
    int2 *items = (int2 *)(up.data() + sizeof(WalkArgs) + 16);
    for (int64_t k = 0; k < nseg; ++k) items[k] = make_int2(0, (int)(q0 + k));
    if ((e = scr.put(scr.owner, d_items, up.data(), up.size())) != cudaSuccess) {
        err = std::string("walker segments: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    SegArgs g{};
    g.args = (const WalkArgs *)d_items;
    g.base = (const int32_t *)(d_items + sizeof(WalkArgs));
    g.items = (const int2 *)(d_items + sizeof(WalkArgs) + 16);
    g.nitems = nseg;
    g.rec[0] = rec;
    g.rec[1] = rec + nseg;
    g.ops = (char *)(rec + 2 * nseg);
    g.xps = (int64_t *)(g.ops + nseg * kSegOps);
    g.gdir = gdir;
    launch_segments(g, a.wide != 0, grid, st);
    *launches += 2;
    std::vector<SegRec> h((size_t)nseg);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = scr.get(scr.owner, h.data(), g.rec[0], sizeof(SegRec) * (size_t)nseg)) != cudaSuccess) {
        err = std::string("walker segments: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    std::vector<int64_t> off;
    int64_t *S = host_state;
    for (int64_t k = nseg - 1; k >= 0 && !S[kStDone]; --k) {
        const SegRec &r = h[(size_t)k];
        if (!r.valid || r.er != S[kStR] || r.ec != S[kStC] || r.est != S[kStState] || r.val != a.score - S[kStSuffix]) break;
        off.push_back(S[kStNOps]);
        off.push_back(S[kStNXp]);
        S[kStR] = r.xr;
        S[kStC] = r.xc;
        S[kStState] = r.xst;
        S[kStNOps] += r.nops;
        S[kStNXp] += r.nxp;
        S[kStSuffix] += r.val - r.xval;
        if (r.done) {
            S[kStDone] = 1;
            S[kStStartR] = r.sr;
            S[kStStartC] = r.sc;
        }
    }
    *taken = (int64_t)off.size() / 2;
    if (*taken == 0) return SWB_OK;
    if (S[kStNOps] > in.ops_cap || S[kStNXp] > in.xp_cap) {
        err = "traceback output larger than its buffers";
        return SWB_ECUDA;
    }
    if ((e = scr.put(scr.owner, d_off, off.data(), sizeof(int64_t) * off.size())) != cudaSuccess) {
        err = std::string("walker segments: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    seg_copy_kernel<<<(unsigned)*taken, 128, 0, st>>>(g.rec[0], g.ops, g.xps, nseg - 1, d_off, in.ops, in.xps);
    *launches += 1;
    if ((e = cudaGetLastError()) != cudaSuccess) {
        err = std::string("walker segments: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    return SWB_OK;
}

int walk_region(cudaStream_t st, int sms, const WalkInputs &in, int64_t *host_state, const Scratch &scr,
                std::string &err, int32_t *launches) {
    const WalkArgs a = to_args(in);
    cudaError_t e;
    const int64_t cap = 4LL * std::max(1, sms);  // blocks per round: one wave at four CTAs per SM
    // as large as segments need it, so that it stays where it is, or without them
    bool segments = host_state[kStR] >= kSegPairMin * (int64_t)a.br;
    uint32_t *gdir = nullptr;
    if (segments) {
        gdir = (uint32_t *)scr.ensure(scr.owner, kScrGdir,
                                      sizeof(uint32_t) * (size_t)(std::max(cap, walk_graph_ctas(sms)) * kBlockWords));
        if (!gdir) cudaGetLastError();
        segments = gdir != nullptr;
    }
    if (!gdir) gdir = (uint32_t *)scr.ensure(scr.owner, kScrGdir, sizeof(uint32_t) * (size_t)(cap * kBlockWords));
    int64_t *d_blk = (int64_t *)scr.ensure(scr.owner, kScrBlk, sizeof(int64_t) * 2 * (size_t)cap);
    int32_t *d_err = (int32_t *)scr.ensure(scr.owner, kScrWalkErr, sizeof(int32_t));
    if (!gdir || !d_blk || !d_err) {
        err = "walker buffers: out of device memory";
        return SWB_ENOMEM;
    }
    if ((e = cudaMemsetAsync(d_err, 0, sizeof(int32_t), st)) != cudaSuccess ||
        (e = scr.put(scr.owner, in.dstate, host_state, sizeof(int64_t) * kStN)) != cudaSuccess) {
        err = std::string("walker state: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    std::vector<int64_t> blk;
    std::vector<int32_t> map;
    // a pair of many blocks: segments at once as long as they continue the path, a
    // corridor round where they do not
    for (int round = 0; round < (1 << 26); ++round) {
        if (segments && !host_state[kStDone] && host_state[kStR] >= kSegPairMin * (int64_t)a.br) {
            int64_t taken = 0;
            const int rc = walk_pair_segments(st, sms, in, a, host_state, gdir, scr, err, launches, &taken);
            if (rc != SWB_OK) return rc;
            segments = taken >= 0;
            if (taken > 0 && (e = scr.put(scr.owner, in.dstate, host_state, sizeof(int64_t) * kStN)) != cudaSuccess) {
                err = std::string("walker state: ") + cudaGetErrorString(e);
                return SWB_ECUDA;
            }
            if (taken >= kSegPairMin) continue;
        }
        const int64_t r = host_state[kStR], c = host_state[kStC];
        if (host_state[kStDone] || host_state[kStErr] || r < in.rr0 || c < in.cc0) break;
        int64_t bi0, bj0, mh, mw;
        predict_corridor(in, r, c, cap, blk, bi0, bj0, mh, mw, map);
        const int64_t nblk = (int64_t)blk.size() / 2;
        int32_t *d_map = (int32_t *)scr.ensure(scr.owner, kScrMap, sizeof(int32_t) * map.size());
        if (!d_map) {
            err = "walker buffers: out of device memory";
            return SWB_ENOMEM;
        }
        if ((e = scr.put(scr.owner, d_blk, blk.data(), sizeof(int64_t) * blk.size())) != cudaSuccess ||
            (e = scr.put(scr.owner, d_map, map.data(), sizeof(int32_t) * map.size())) != cudaSuccess) {
            err = std::string("walker corridor: ") + cudaGetErrorString(e);
            return SWB_ECUDA;
        }
        if (a.wide) precompute_kernel<true><<<(unsigned)nblk, kThreadsWide, 0, st>>>(a, d_blk, nblk, gdir, d_err);
        else precompute_kernel<false><<<(unsigned)nblk, kThreads, 0, st>>>(a, d_blk, nblk, gdir, d_err);
        corridor_walk_kernel<<<1, 32, kDirTileBytes, st>>>(a, gdir, d_map, bi0, bj0, mh, mw, d_err);
        *launches += 2;
        if ((e = cudaGetLastError()) != cudaSuccess ||
            (e = scr.get(scr.owner, host_state, in.dstate, sizeof(int64_t) * kStN)) != cudaSuccess) {
            err = std::string("walker: ") + cudaGetErrorString(e);
            return SWB_ECUDA;
        }
        if (host_state[kStR] == r && host_state[kStC] == c && !host_state[kStDone] && !host_state[kStErr]) {
            err = "walker: no progress through the current block";
            return SWB_ECUDA;
        }
    }
    if (host_state[kStErr]) {
        err = "walker: inconsistent direction data";
        return SWB_ECUDA;
    }
    return SWB_OK;
}

int walk_cells(cudaStream_t st, int sms, const WalkInputs &whole, const std::vector<WalkInputs> &cells, int64_t kr,
               int64_t kc, int64_t *host_state, const Scratch &scr, std::string &err, int32_t *launches) {
    WalkInputs base = whole;
    base.br = kBR;
    const WalkArgs a = to_args(base);
    const int64_t cap = 4LL * std::max(1, sms);
    std::vector<WalkArgs> regs(cells.size());
    std::unordered_map<int64_t, int32_t> find;  // (cell row, cell column) -> region
    for (size_t q = 0; q < cells.size(); ++q) {
        regs[q] = to_args(cells[q]);
        find.emplace((cells[q].rr0 / kr << 32) | (cells[q].cc0 / kc), (int32_t)q);
    }
    cudaError_t e;
    uint32_t *gdir = (uint32_t *)scr.ensure(scr.owner, kScrGdir, sizeof(uint32_t) * (size_t)(cap * kBlockWords));
    WalkArgs *d_regs = (WalkArgs *)scr.ensure(scr.owner, kScrSegItems, sizeof(WalkArgs) * regs.size());
    int32_t *d_err = (int32_t *)scr.ensure(scr.owner, kScrWalkErr, sizeof(int32_t));
    if (!gdir || !d_regs || !d_err) {
        err = "walker buffers: out of device memory";
        return SWB_ENOMEM;
    }
    if ((e = cudaMemsetAsync(d_err, 0, sizeof(int32_t), st)) != cudaSuccess ||
        (e = scr.put(scr.owner, d_regs, regs.data(), sizeof(WalkArgs) * regs.size())) != cudaSuccess ||
        (e = scr.put(scr.owner, base.dstate, host_state, sizeof(int64_t) * kStN)) != cudaSuccess) {
        err = std::string("walker cells: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    std::vector<int64_t> blk;
    std::vector<int32_t> map, reg;
    std::vector<char> up;
    for (int round = 0; round < (1 << 26); ++round) {
        const int64_t r = host_state[kStR], c = host_state[kStC];
        if (host_state[kStDone] || host_state[kStErr] || r < 0 || c < 0) break;
        if (find.find((r / kr << 32) | (c / kc)) == find.end()) break;  // the path left the cells
        int64_t bi0, bj0, mh, mw;
        predict_corridor(base, r, c, cap, blk, bi0, bj0, mh, mw, map);
        // blocks of cells that are there, their regions and their slots
        std::vector<int32_t> slot(blk.size() / 2, -1);
        int32_t kept = 0;
        reg.clear();
        for (size_t b = 0; b < slot.size(); ++b) {
            const auto it = find.find((blk[2 * b] / kr << 32) | (blk[2 * b + 1] / kc));
            if (it == find.end()) continue;
            blk[2 * (size_t)kept] = blk[2 * b];
            blk[2 * (size_t)kept + 1] = blk[2 * b + 1];
            reg.push_back(it->second);
            slot[b] = kept++;
        }
        for (int32_t &v : map)
            if (v >= 0) v = slot[(size_t)v];
        const size_t nb = sizeof(int64_t) * 2 * (size_t)kept, nr = sizeof(int32_t) * (size_t)kept,
                     nm = sizeof(int32_t) * map.size();
        up.resize(nb + nr + nm);
        std::memcpy(up.data(), blk.data(), nb);
        std::memcpy(up.data() + nb, reg.data(), nr);
        std::memcpy(up.data() + nb + nr, map.data(), nm);
        char *d_up = (char *)scr.ensure(scr.owner, kScrMap, up.size());
        if (!d_up) {
            err = "walker buffers: out of device memory";
            return SWB_ENOMEM;
        }
        if ((e = scr.put(scr.owner, d_up, up.data(), up.size())) != cudaSuccess) {
            err = std::string("walker cells: ") + cudaGetErrorString(e);
            return SWB_ECUDA;
        }
        const int64_t *d_blk = (const int64_t *)d_up;
        const int32_t *d_reg = (const int32_t *)(d_up + nb), *d_map = (const int32_t *)(d_up + nb + nr);
        if (a.wide) precompute_cells_kernel<true><<<(unsigned)kept, kThreadsWide, 0, st>>>(d_regs, d_blk, d_reg, kept, gdir, d_err);
        else precompute_cells_kernel<false><<<(unsigned)kept, kThreads, 0, st>>>(d_regs, d_blk, d_reg, kept, gdir, d_err);
        corridor_walk_kernel<<<1, 32, kDirTileBytes, st>>>(a, gdir, d_map, bi0, bj0, mh, mw, d_err);
        *launches += 2;
        if ((e = cudaGetLastError()) != cudaSuccess ||
            (e = scr.get(scr.owner, host_state, base.dstate, sizeof(int64_t) * kStN)) != cudaSuccess) {
            err = std::string("walker cells: ") + cudaGetErrorString(e);
            return SWB_ECUDA;
        }
        if (host_state[kStR] == r && host_state[kStC] == c && !host_state[kStDone] && !host_state[kStErr]) {
            err = "walker: no progress through the current block";
            return SWB_ECUDA;
        }
    }
    if (host_state[kStErr]) {
        err = "walker: inconsistent direction data";
        return SWB_ECUDA;
    }
    return SWB_OK;
}

int64_t walk_batch_ctas(int sms, int64_t n) { return std::max<int64_t>(1, std::min<int64_t>(n, 8LL * std::max(1, sms))); }
size_t walk_batch_dir_bytes(int sms, int64_t n) {
    return sizeof(uint32_t) * (size_t)kBlockWords * (size_t)walk_batch_ctas(sms, n);
}

int walk_batch(cudaStream_t st, int sms, const WalkInputs *in, int64_t n, void *d_args, int64_t *d_states,
               uint64_t seg_bytes, int64_t *host_states, const Scratch &scr, std::string &err, int32_t *launches) {
    if (n <= 0) return SWB_OK;
    std::vector<WalkArgs> args((size_t)n);
    std::vector<int64_t> rows((size_t)n);
    for (int64_t i = 0; i < n; ++i) {
        args[(size_t)i] = to_args(in[i]);
        args[(size_t)i].st = d_states + i * kStN;
        rows[(size_t)i] = in[i].m;
    }
    const bool wide = args[0].wide != 0;
    cudaError_t e;
    const int64_t grid = walk_batch_ctas(sms, n);
    if ((e = scr.put(scr.owner, d_args, args.data(), sizeof(WalkArgs) * (size_t)n)) != cudaSuccess ||
        (e = scr.put(scr.owner, d_states, host_states, sizeof(int64_t) * kStN * (size_t)n)) != cudaSuccess) {
        err = std::string("batched walker set-up: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    SegArgs g{};
    std::vector<int32_t> base, items;
    int64_t nseg = seg_plan(rows.data(), n, seg_bytes, base, items);
    const int64_t sgrid = std::min<int64_t>(walk_graph_ctas(sms), nseg);
    auto blocks = [&](int64_t ctas) {
        return (uint32_t *)scr.ensure(scr.owner, kScrGdir, sizeof(uint32_t) * (size_t)(ctas * kBlockWords));
    };
    // segments and walk run one after the other on the same direction blocks; where
    // there is no memory for segments, the pairs are walked in one piece
    uint32_t *gdir = nullptr;
    SegRec *rec = nullptr;
    int32_t *d_items = nullptr;
    if (nseg > 0) {
        rec = (SegRec *)scr.ensure(scr.owner, kScrSegRec, seg_scratch_bytes(nseg));
        d_items = (int32_t *)scr.ensure(scr.owner, kScrSegItems, sizeof(int32_t) * (items.size() + base.size()));
        if (rec && d_items) gdir = blocks(std::max(grid, sgrid));
        if (!gdir) {
            cudaGetLastError();
            nseg = 0;
        }
    }
    if (!gdir && !(gdir = blocks(grid))) {
        err = "walker buffers: out of device memory";
        return SWB_ENOMEM;
    }
    if (nseg > 0) {
        std::vector<int32_t> up(items);
        up.insert(up.end(), base.begin(), base.end());
        if ((e = scr.put(scr.owner, d_items, up.data(), sizeof(int32_t) * up.size())) != cudaSuccess) {
            err = std::string("batched walker segments: ") + cudaGetErrorString(e);
            return SWB_ECUDA;
        }
        g.args = (const WalkArgs *)d_args;
        g.items = (const int2 *)d_items;
        g.nitems = nseg;
        g.base = d_items + items.size();
        g.rec[0] = rec;
        g.rec[1] = rec + nseg;
        g.ops = (char *)(rec + 2 * nseg);
        g.xps = (int64_t *)(g.ops + nseg * kSegOps);
        g.gdir = gdir;
        launch_segments(g, wide, sgrid, st);
        *launches += 2;
    }
    if (wide) walk_batch_kernel<true><<<(unsigned)grid, kThreadsWide, 0, st>>>((const WalkArgs *)d_args, n, gdir, g);
    else walk_batch_kernel<false><<<(unsigned)grid, kThreads, 0, st>>>((const WalkArgs *)d_args, n, gdir, g);
    *launches += 1;
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = scr.get(scr.owner, host_states, d_states, sizeof(int64_t) * kStN * (size_t)n)) != cudaSuccess) {
        err = std::string("batched walker: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    for (int64_t i = 0; i < n; ++i)
        if (host_states[i * kStN + kStErr] || !host_states[i * kStN + kStDone]) {
            err = "batched walker: inconsistent direction data";
            return SWB_ECUDA;
        }
    return SWB_OK;
}

int pack_results(cudaStream_t st, const void *d_args, int64_t n, const int64_t *host_states, const int64_t *ends,
                 std::vector<int64_t> &offs, int64_t *ops_bytes, int64_t *n_xps, char **d_ops, swb_xpoint **d_xps,
                 const Scratch &scr, std::string &err) {
    offs.resize((size_t)(4 * n));
    int64_t po = 0, px = 0;
    for (int64_t i = 0; i < n; ++i) {
        const int64_t *S = host_states + i * kStN;
        int64_t *o = offs.data() + 4 * i;
        o[0] = po;
        o[1] = px;
        o[2] = ends[2 * i];
        o[3] = ends[2 * i + 1];
        po += S[kStNOps];
        px += S[kStNXp] + 2;
    }
    *ops_bytes = po;
    *n_xps = px;
    int64_t *d_off = (int64_t *)scr.ensure(scr.owner, kScrSegOff, sizeof(PackOff) * (size_t)n);
    *d_ops = (char *)scr.ensure(scr.owner, kScrOps, (size_t)po + 1);
    *d_xps = (swb_xpoint *)scr.ensure(scr.owner, kScrXps, sizeof(swb_xpoint) * (size_t)px);
    cudaError_t e;
    if (!d_off || !*d_ops || !*d_xps) {
        err = "result buffers: out of device memory";
        return SWB_ENOMEM;
    }
    static_assert(sizeof(PackOff) == 4 * sizeof(int64_t), "PackOff layout");
    if ((e = scr.put(scr.owner, d_off, offs.data(), sizeof(PackOff) * (size_t)n)) == cudaSuccess) {
        pack_results_kernel<<<(unsigned)n, 256, 0, st>>>((const WalkArgs *)d_args, (const PackOff *)d_off, *d_ops, *d_xps);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        err = std::string("batched results: ") + cudaGetErrorString(e);
        return SWB_ECUDA;
    }
    return SWB_OK;
}

void pack_walk_args(const WalkInputs *in, int64_t n, int64_t *d_states, void *dst) {
    WalkArgs *out = (WalkArgs *)dst;
    for (int64_t i = 0; i < n; ++i) {
        WalkArgs a = to_args(in[i]);
        a.st = d_states + i * kStN;
        std::memcpy(out + i, &a, sizeof a);
    }
}

cudaError_t walk_graph_enqueue(const GraphHdr *d_hdr, bool wide, bool segments, int sms, int64_t max_pairs,
                               int64_t max_units, cudaStream_t st) {
    const int64_t p = std::max<int64_t>(1, max_pairs);
    walk_graph_init_kernel<<<(unsigned)std::min<int64_t>(std::max(1, sms), (p + 255) / 256), 256, 0, st>>>(d_hdr);
    if (segments) {  // the guess writes the second records, the next round the first
        const unsigned sgrid = (unsigned)std::min<int64_t>(walk_graph_ctas(sms), std::max<int64_t>(1, max_units));
        if (wide) {
            seg_graph_kernel<true, true><<<sgrid, kThreadsWide, 0, st>>>(d_hdr, 0);
            seg_graph_kernel<true, false><<<sgrid, kThreadsWide, 0, st>>>(d_hdr, 1);
        } else {
            seg_graph_kernel<false, true><<<sgrid, kThreads, 0, st>>>(d_hdr, 0);
            seg_graph_kernel<false, false><<<sgrid, kThreads, 0, st>>>(d_hdr, 1);
        }
    }
    const unsigned grid = (unsigned)std::min<int64_t>(walk_graph_ctas(sms), p);
    if (wide) walk_graph_kernel<true><<<grid, kThreadsWide, 0, st>>>(d_hdr);
    else walk_graph_kernel<false><<<grid, kThreads, 0, st>>>(d_hdr);
    return cudaGetLastError();
}

int64_t seg_plan(const int64_t *rows, int64_t n, uint64_t max_bytes, std::vector<int32_t> &base,
                 std::vector<int32_t> &items) {
    base.assign((size_t)n, -1);
    items.clear();
    int64_t total = 0;
    for (int64_t p = 0; p < n; ++p) total += (rows[p] + kBR - 1) / kBR;
    // Segments pay even where the pairs alone fill
    // the GPU: few are walked twice, and none is left over at the end (1,000 long
    // pairs of the 100,000-pair batch: 6.4 ms, against about 15 ms walked pair by pair).
    if (total > kSegMax || seg_scratch_bytes(total) > max_bytes) return 0;
    int32_t seg = 0;
    for (int64_t p = 0; p < n; ++p) {
        const int32_t k = (int32_t)((rows[p] + kBR - 1) / kBR);
        if (k < kSegMin) continue;
        base[(size_t)p] = seg;
        for (int32_t q = 0; q < k; ++q) {
            items.push_back((int32_t)p);
            items.push_back(q);
        }
        seg += k;
    }
    return seg;
}

size_t seg_scratch_bytes(int64_t nseg) {
    return (size_t)nseg * (2 * sizeof(SegRec) + kSegOps + sizeof(int64_t) * 4 * kSegXps);
}

uint64_t seg_pair_bytes(int64_t rows) {
    const int64_t k = (rows + kBR - 1) / kBR;
    return k < kSegMin ? 0 : (uint64_t)seg_scratch_bytes(k);
}

int64_t seg_window() { return kSegWindow; }

int64_t walk_graph_ctas(int sms) { return 8LL * std::max(1, sms); }

size_t walk_args_bytes() { return sizeof(WalkArgs); }

int state_slots() { return kStN; }
int slot_r() { return kStR; }
int slot_c() { return kStC; }
int slot_state() { return kStState; }
int slot_nops() { return kStNOps; }
int slot_nxp() { return kStNXp; }
int slot_done() { return kStDone; }
int slot_err() { return kStErr; }
int slot_start_r() { return kStStartR; }
int slot_start_c() { return kStStartC; }
int block_rows() { return kBR; }
int block_cols() { return kBC; }

}  // namespace tb
}  // namespace swb

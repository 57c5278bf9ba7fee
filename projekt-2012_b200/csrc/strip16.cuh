// strip16.cuh -- the scoring strip in packed 16-bit lanes: two cells per
// instruction within one pair, with exact 32-bit results.
//
// Same recurrence and the same strips, hand-off entries, special rows and
// columns as stage1_core.cuh (src/FindAlignment.cuh:50-104 of the reference);
// a strip of 64*RH rows runs on one warp whose 32-bit registers each hold two
// rows' values: lane l's low half rows [l*RH, (l+1)*RH) of the strip and its
// high half the same rows 32*RH further down.  The warp is a wavefront of 64
// virtual lanes: at step k the low half of lane l computes column k - l and the
// high half column k - l - 32.  One rotating shuffle moves (H, F) of both halves
// to the next lane; lane 31 sends its low half to lane 0's high half and the
// next column's top boundary to lane 0's low half.
//
// Values.  A cell's H + open, E and F are held as base + a 16-bit offset, base
// a 32-bit number of the whole warp that is moved when the offsets near the ends
// of their range; everything stored outside the warp is the 32-bit value again.
// Offsets are exact integers, so results are those of the 32-bit recurrence as
// long as every value of the warp fits its window:
//   * spread: for any two cells of the matrix |H - H'| <= (rows + columns between
//     them) * (match + e) + 2 |open| with e = min(|open|, |extend|) (extend the
//     better cell's alignment by gaps; trim the other's), so cells of one warp
//     (64 RH rows, about 130 columns apart) lie within a few thousand of each
//     other.  The caller checks that bound (strip16_fits), and every 32 steps
//     each lane checks its bottom row against the window, the margin of the
//     rows and columns in between included; a span that does not fit sets
//     kErrRange, and the host scores the pair in 32 bits.
//   * the zero floor: with base = 0 the relu is the recurrence's.  With base > 0
//     the window keeps every H above base, where neither floor has an effect
//     (flooring t at base changes no H >= base, and F and E of the next cell are
//     at least H + open either way).
//
// What bounds it: the ALU pipe, where each packed op (and LOP3, PRMT) alone issues at
// 64 lanes per SM and cycle: 6 per row pair (PRMT score, E, t, t + open, H, F'), which
// together take 10.8 cycles per warp and sub-partition for 64 cells
// (swb_probe_packed_peak), against 10.3 for 32 cells of the 32-bit step.
//
// Best cell.  The step itself does not look for it.  Before each run of 32 steps
// the warp asks whether any cell of the run could reach the best H known (bottom
// rows + the bound above, and the row above where a given border need not keep the
// bound): if not, the steps run without a column maximum.  If
// so, the state is kept in shared memory, the steps fold a running maximum, and
// only when that reaches the best known does the warp remember the run (instead
// of the ones remembered before, which it beats: along an alignment path that is
// every time).  Remembered runs are done again with exact cells and tie keys only
// when they still hold the best when the strip ends, or when there are too many
// of the same value.
#pragma once

#include "stage1_core.cuh"

namespace swb {
namespace {

constexpr int32_t kErrRange = kStage1Range;  // a 16-bit window did not hold: score in 32 bits

__device__ __forceinline__ int32_t half16(uint32_t v, int h) { return (int32_t)(int16_t)(uint16_t)(v >> (16 * h)); }
__device__ __forceinline__ uint32_t dup16(int32_t v) { return (uint32_t)(uint16_t)(int16_t)v * 0x00010001u; }
__device__ __forceinline__ int32_t max16(uint32_t v) { return max(half16(v, 0), half16(v, 1)); }

// Lane state: everything a step reads and writes besides the column words.
template <int RH>
struct Lane2 {
    uint32_t HO[RH];    // H + open of the previous column (offsets)
    uint32_t E[RH];     // E of the previous column
    uint32_t inHO, inF; // from the virtual lane above: H + open of its last row, F of my row 0
    uint32_t hod;       // H + open above my row 0 at the previous column
};

constexpr int kRun = 32;       // steps between refills: a lane per column
// Steps unrolled in a loop's body.  A run walks through its body's code four to
// sixteen times, so what it costs is instruction fetch: with 8 steps of 16 row
// pairs unrolled in every variant the 400 kbp pair's store pass took 147 ms, with
// 4, and 2 in the special-column and edge runs, 78 ms; 8 row pairs run 5% faster
// with 8 steps than with 4.
template <int RH>
struct Sub {
    static constexpr int plain = RH <= 8 ? 8 : 4, edge = RH <= 4 ? 4 : 2;
};
constexpr int kColRing = 128;  // column values kept: 63 behind (the high half of lane 31), 63 ahead

// Runs kept at once (the one in progress included).  Eight instead of three 256-row
// strips' runs: unrelated 15 kbp pair, stage 1 1.59 -> 1.54 ms.
template <int RH>
constexpr int kKept = RH <= 4 ? 8 : (RH <= 8 ? 3 : 2);

// A warp's shared memory.
template <int RH>
struct WarpMem {
    uint4 save[kKept<RH>][(RH + 1) / 2 + 1][32];  // lane states before the kept runs: HO, E of two rows each; inHO, inF, hod
    uint4 spec[(RH + 1) / 2][32];                 // HO, E of a special column's rows, per lane; of all rows during a rerun
    int2 stage[kRun];                             // lane 31's last rows (H + open, F) of the last run (special rows)
    uint32_t ring[kRun + 1];                      // row above (H + open | F << 16) of the next step's column, per step
    uint32_t sring[kKept<RH>][kRun];              // the same of the kept runs
    uint32_t col[kColRing + kRun + 1];            // column values; the first kRun kept twice, so that a run is contiguous
    int32_t kept_k[kKept<RH>], kept_base[kKept<RH>], kept_val[kKept<RH>];
    // the warp's best cell
    int32_t best_ho, best_valid;
    uint64_t best_key;
    int64_t best_row, best_col;
};

// Once per launch: no best cell yet, and column values that are valid codes
// (halves outside the matrix read entries that no column was kept in).
template <int RH>
__device__ __forceinline__ void init_warp(WarpMem<RH> *w, int lane, int32_t open) {
    for (int i = lane; i < kColRing + kRun; i += 32) w->col[i] = 0;
    if (lane == 0) {
        w->best_ho = open + 1;  // only H >= 1 is recorded
        w->best_valid = 0;
        w->best_key = ~0ULL;
        w->best_row = 0;
        w->best_col = 0;
    }
    __syncwarp();
}

// A hand-off entry {H + open | F << 16 (offsets), tag, base, tag}: as in
// stage1_core.cuh each 8-byte half carries the writing strip's tag.
__device__ __forceinline__ void st_hand(int4 *p, uint32_t hf, int32_t base, int32_t tag) {
    asm volatile("st.volatile.global.v4.s32 [%0], {%1,%2,%3,%2};" ::"l"(p), "r"(hf), "r"(tag), "r"(base));
}

// Packed scoring constants.
struct Consts2 {
    uint32_t open2, ext2, gx2, mt1p2, mm12;
};
__device__ __forceinline__ Consts2 consts2(int32_t open, int32_t ext, int32_t gx, int32_t mt1, int32_t mm1) {
    Consts2 c;
    c.open2 = dup16(open);
    c.ext2 = dup16(ext);
    c.gx2 = dup16(gx);
    c.mt1p2 = dup16(mt1 + 1);
    c.mm12 = dup16(mm1);
    return c;
}

// Both halves' substitution scores (minus open) of one row.  CMP: column and row
// bytes shifted left by 6, so that unequal ones differ by at least 64 and
// max(~(ra ^ c) + mt1 + 1, mm1) is mt1 for equal bytes and mm1 otherwise (the
// caller checks mt1 - mm1 <= 64).
template <bool TAB>
__device__ __forceinline__ uint32_t score2(uint32_t cA, uint32_t cB, uint32_t ra, const Consts2 &c) {
    if (TAB) return (uint32_t)prmt(cA, cB, ra);
    return __viaddmax_s16x2(~(ra ^ cA), c.mt1p2, c.mm12);
}

// How a lane's registers leave a step.
struct Turn {
    uint32_t selH, selF;  // PRMT selectors of H and F toward the next lane (lane 31: the ring's entry comes in)
    bool hand;            // lane 31 of a strip with a strip below: hand the bottom row down
    bool keep;            // lane 31 of a strip whose rows are stored
    int32_t tag, base;
    int spec;             // SC: the step of the unrolled ones after which my rows go to the special column
};

// One step.  ca, cb: this step's column values of the low and high half (loaded
// from shared memory by each lane, so they wait for no shuffle); rv: the next
// column's row above; hb: hand-off entry of lane 31's column, st: its place in the
// stage.  TRACK: fold t + open of every row into mx (packed maxima).  EDGE: lane
// 31's column may be outside [0, n): `inside` says.  PRED: halves outside [0, n)
// keep their values: mask has 0xFFFF in each half that is inside.  PRED with ROWS: mx
// takes only the rectangle's rows: bits i and 16 + i of rows for row i of the halves.
//
// A warp issues in order, and alone on its scheduler it is bound by latencies.
// Phase 1 (scores, E, t: 8 issue cycles a row) needs only the previous step's H
// and E and covers the shuffle of H and F from the lane above; phase 2 is the F
// chain, whose two ops a row issue in the 4 cycles that one of them takes.
enum : int { kPlain = 0, kEdge = 1, kPred = 2, kPredRows = 3 };
template <int RH, bool TAB, bool TRACK, int MODE, bool STORES, bool SC>
__device__ __forceinline__ void step2(Lane2<RH> &L, const uint32_t *ra, const Consts2 &c, uint32_t ca, uint32_t cb,
                                      uint32_t rv, int4 *hb, int2 *st, uint4 (*sp)[32], int v, int lane, const Turn &t,
                                      bool inside, uint32_t mask, uint32_t rows, uint32_t &mx) {
    constexpr bool PRED = MODE == kPred || MODE == kPredRows, ROWS = MODE == kPredRows;
    uint32_t to[RH];
    if (!TAB) ca = cb * 65536u + ca;
    uint32_t hod = L.hod;
#pragma unroll
    for (int i = 0; i < RH; ++i) {
        const uint32_t s1 = score2<TAB>(ca, cb, ra[i], c);
        const uint32_t e = __viaddmax_s16x2(L.E[i], c.ext2, L.HO[i]);
        to[i] = __vadd2(__viaddmax_s16x2_relu(hod, s1, e), c.open2);
        hod = L.HO[i];
        L.E[i] = PRED ? ((e & mask) | (L.E[i] & ~mask)) : e;
    }
    if (TRACK) {
        uint32_t m = PRED ? 0x80008000u : mx;
        if (ROWS) {
#pragma unroll
            for (int i = 0; i < RH; ++i) {
                const uint32_t in = ((rows >> i) & 0x00010001u) * 0xFFFFu;
                m = __vmaxs2(m, (to[i] & in) | (0x80008000u & ~in));
            }
        } else {
#pragma unroll
            for (int i = 0; i + 1 < RH; i += 2) m = __vimax3_s16x2(m, to[i], to[i + 1]);
            if (RH & 1) m = __vmaxs2(m, to[RH - 1]);
        }
        mx = PRED ? __vmaxs2(mx, (m & mask) | (0x80008000u & ~mask)) : m;
    }
    uint32_t f = L.inF, flast = 0;
#pragma unroll
    for (int i = 0; i < RH; ++i) {
        const uint32_t ho = __viaddmax_s16x2(f, c.open2, to[i]);
        flast = f;
        f = __viaddmax_s16x2(f, c.gx2, to[i]);
        L.HO[i] = PRED ? ((ho & mask) | (L.HO[i] & ~mask)) : ho;
    }
    const uint32_t oF = (uint32_t)prmt(rv, f, t.selF);
    const uint32_t oHO = (uint32_t)prmt(rv, L.HO[RH - 1], t.selH);
    const int src = (lane + 31) & 31;
    L.hod = L.inHO;
    L.inF = __shfl_sync(0xffffffffu, oF, src);
    L.inHO = __shfl_sync(0xffffffffu, oHO, src);
    // the strip below takes lane 31's high half: both values in one word, with the
    // base that its offsets are relative to
    if (t.hand && (MODE == kPlain || inside)) st_hand(hb, (uint32_t)prmt(L.HO[RH - 1], f, 0x7632u), t.base, t.tag);
    if (STORES && t.keep) *st = make_int2((int32_t)L.HO[RH - 1], (int32_t)flast);
    if (SC && t.spec == v) {
#pragma unroll
        for (int i = 0; i < RH; i += 2) {
            const int i1 = i + 1 < RH ? i + 1 : i;
            sp[i / 2][lane] = make_uint4(L.HO[i], L.HO[i1], L.E[i], L.E[i1]);
        }
    }
}

// The rows of a lane (first rows r and r + 32 RH) above row m, as step2 takes them.
template <int RH>
__device__ __forceinline__ uint32_t rows_in(int64_t r, int64_t m) {
    const int64_t l = m - r, h = l - 32 * RH;
    const uint32_t nl = (uint32_t)max((int64_t)0, min(l, (int64_t)RH)), nh = (uint32_t)max((int64_t)0, min(h, (int64_t)RH));
    return ((1u << nl) - 1u) | (((1u << nh) - 1u) << 16);
}

// 0xFFFF in each half whose column at step k lies in [0, n).
__device__ __forceinline__ uint32_t active2(int32_t k, int lane, int32_t n) {
    const int32_t jl = k - lane, jh = jl - 32;
    return ((jl >= 0 && jl < n) ? 0x0000FFFFu : 0u) | ((jh >= 0 && jh < n) ? 0xFFFF0000u : 0u);
}

template <int RH>
__device__ __forceinline__ void put_state(WarpMem<RH> *w, int q, int lane, const Lane2<RH> &L) {
#pragma unroll
    for (int i = 0; i + 1 < RH; i += 2) w->save[q][i / 2][lane] = make_uint4(L.HO[i], L.HO[i + 1], L.E[i], L.E[i + 1]);
    if (RH & 1) w->save[q][RH / 2][lane] = make_uint4(L.HO[RH - 1], 0, L.E[RH - 1], 0);
    w->save[q][(RH + 1) / 2][lane] = make_uint4(L.inHO, L.inF, L.hod, 0);
}

// What column c is read as: the table word (TAB) or the byte; and its column value.
template <bool TAB>
__device__ __forceinline__ uint32_t read_col(const uint32_t *ctab, const uint8_t *cols, int32_t c) {
    return TAB ? ctab[c] : (uint32_t)cols[c];
}
template <bool TAB>
__device__ __forceinline__ uint32_t col_value(uint32_t v) {
    return TAB ? v : v << 6;
}
template <bool TAB>
__device__ __forceinline__ uint32_t col2(const uint32_t *ctab, const uint8_t *cols, int32_t c) {
    return col_value<TAB>(read_col<TAB>(ctab, cols, c));
}

// The loads that are issued a run before their values are used write the very
// registers that are carried around the loop, whatever was in them having been used
// before, and are predicated.  Written as assignments in branches they were given
// registers of their own, and the moves into the carried ones, put right behind the
// loads, waited for each: a refill of a lone warp's 256-row strip took 1000 to 1300
// cycles of a run's 3400, and takes 600 (score only, 61 kbp pair: 4.6 -> 3.75 ms).
__device__ __forceinline__ void ld_hand(int4 &v, bool on, const int4 *p) {
    asm volatile("{.reg .pred p; setp.ne.s32 p, %5, 0; @p ld.volatile.global.v4.s32 {%0,%1,%2,%3}, [%4];}"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
                 : "l"(p), "r"((int)on));
}
template <bool TAB>
__device__ __forceinline__ void ld_col(uint32_t &v, bool on, const uint32_t *ctab, const uint8_t *cols, int32_t c) {
    if (TAB)
        asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p ld.global.u32 %0, [%1];}" : "+r"(v) : "l"(ctab + c), "r"((int)on));
    else
        asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p ld.global.u8 %0, [%1];}" : "+r"(v) : "l"(cols + c), "r"((int)on));
}
__device__ __forceinline__ void ld_best(int32_t &v, const int32_t *p) {
    asm volatile("ld.volatile.global.s32 %0, [%1];" : "+r"(v) : "l"(p));
}

// Row selector (TAB) or code (CMP) of rows r0 + i and r0 + 32 RH + i.
template <int RH, bool TAB>
__device__ __forceinline__ uint32_t row2(const uint8_t *rcode, const uint8_t *rows, int64_t m, int64_t r0) {
    uint32_t sel[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int64_t r = r0 + h * 32 * RH;
        const bool in = r < m;
        if (TAB) {
            // a row past the end takes a table byte's sign in both bytes: a score of
            // open or open - 1, never a match
            const uint32_t q = (in ? (uint32_t)rcode[r] : 8u) + 4u * h;
            sel[h] = in ? (q | ((q | 8u) << 4)) : (q | 8u) * 0x11u;
        } else {
            sel[h] = (in ? (uint32_t)rows[r] : 256u) << 6;
        }
    }
    return TAB ? (sel[0] | (sel[1] << 8)) : (sel[0] | (sel[1] << 16));
}

// Does the kept run of slot q again (L is overwritten), finds the cells that hold
// its maximum and merges the one with the smallest tie key into the warp's best.
template <int RH, bool TAB, bool RAGGED, class A>
__device__ __forceinline__ void rerun(const A &a, WarpMem<RH> *w, Lane2<RH> &L, const uint32_t *ra, const Consts2 &c, int q,
                                      int lane, int64_t r_lane) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i + 1 < RH; i += 2) {
        const uint4 v = w->save[q][i / 2][lane];
        L.HO[i] = v.x;
        L.HO[i + 1] = v.y;
        L.E[i] = v.z;
        L.E[i + 1] = v.w;
    }
    if (RH & 1) {
        const uint4 v = w->save[q][RH / 2][lane];
        L.HO[RH - 1] = v.x;
        L.E[RH - 1] = v.z;
    }
    {
        const uint4 v = w->save[q][(RH + 1) / 2][lane];
        L.inHO = v.x;
        L.inF = v.y;
        L.hod = v.z;
    }
    const int32_t k0 = w->kept_k[q], target = w->kept_val[q] - w->kept_base[q], n = (int32_t)a.n;
    const Turn t{lane == 31 ? 0x5410u : 0x7654u, lane == 31 ? 0x5432u : 0x7654u, false, false, 0, 0, 0};
    const uint32_t rows = RAGGED ? rows_in<RH>(r_lane, a.m) : 0u;
    uint64_t bkey = ~0ULL;
    int64_t brow = 0, bcol = 0;
#pragma unroll 1
    for (int u = 0; u < kRun; ++u) {
        const uint32_t mask = active2(k0 + u, lane, n);
        uint32_t mx = 0x80008000u;
        const uint32_t ca = (mask & 1u) ? col2<TAB>(a.ctab, a.cols, k0 + u - lane) : 0u;
        const uint32_t cb = (mask >> 16) ? col2<TAB>(a.ctab, a.cols, k0 + u - lane - 32) : 0u;
        step2<RH, TAB, true, RAGGED ? kPredRows : kPred, false, false>(L, ra, c, ca, cb, w->sring[q][u], nullptr, nullptr, nullptr, 0, lane, t,
                                                  false, mask, rows, mx);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            if (half16(mx, h) != target || !((mask >> (16 * h)) & 1u)) continue;
            const int64_t r0 = r_lane + h * 32 * RH;
            const int64_t j = (int64_t)(k0 + u - lane - 32 * h);
            uint32_t hold = 0;
#pragma unroll
            for (int i = 0; i < RH; ++i) hold |= (half16(L.HO[i], h) == target ? 1u : 0u) << i;
            for (; hold; hold &= hold - 1) {
                const int64_t r = r0 + __ffs(hold) - 1;
                if (r >= a.m) break;
                const uint64_t key = tie_key(a.tie, a.r_origin + r, a.c_origin + j);
                if (key < bkey) {
                    bkey = key;
                    brow = r;
                    bcol = j;
                }
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const uint64_t okey = __shfl_xor_sync(0xffffffffu, bkey, off);
        const int64_t orow = __shfl_xor_sync(0xffffffffu, brow, off);
        const int64_t ocol = __shfl_xor_sync(0xffffffffu, bcol, off);
        if (okey < bkey) {
            bkey = okey;
            brow = orow;
            bcol = ocol;
        }
    }
    if (lane == 0 && bkey != ~0ULL) {
        const int32_t v = w->kept_val[q];
        if (v > w->best_ho || (v == w->best_ho && bkey < w->best_key)) {
            w->best_ho = v;
            w->best_valid = 1;
            w->best_key = bkey;
            w->best_row = brow;
            w->best_col = bcol;
        }
    }
    __syncwarp();
}

// Where a strip's last rows go besides the strip below.
struct Out2 {
    int2 *row[2];  // per half: special row or the rectangle's last row (column 0), or null
};

// Columns lane 31 staged in the run of steps before step k (a lane per step).
template <int RH>
__device__ __forceinline__ void flush2(const WarpMem<RH> *w, int lane, const Out2 &o, int32_t n, int32_t k, int32_t base,
                                       int32_t open) {
    const int2 v = w->stage[lane];
    const int32_t cl = k - kRun + lane - 31, ch = cl - 32;
    if (o.row[0] && cl >= 0 && cl < n)
        o.row[0][cl] = make_int2(half16((uint32_t)v.x, 0) + base - open, half16((uint32_t)v.y, 0) + base);
    if (o.row[1] && ch >= 0 && ch < n)
        o.row[1][ch] = make_int2(half16((uint32_t)v.x, 1) + base - open, half16((uint32_t)v.y, 1) + base);
}

// The row above the strip at column c as a hand-off entry: the strip above's, a
// given top boundary or the matrix edge (relative to H + open of that cell).
template <bool BORDERS, class A>
__device__ __forceinline__ int4 above2(const A &a, int32_t strip, int32_t c) {
    if (strip > 0) return ld_ll(a.hbuf + c);
    if (BORDERS && a.top) {
        const int2 t = a.top[c];
        const int32_t d = max(t.y + a.ext - t.x - a.open, 0);  // F of row 0 above H + open
        return make_int4((int32_t)((uint32_t)min(d, 32767) << 16), 0, t.x + a.open, 0);
    }
    return make_int4((int32_t)((uint32_t)(a.gx - a.open) << 16), 0, a.open, 0);  // H = 0 above the first row
}

// Column c's entry, loaded earlier, as offsets from base (loading it again until
// the strip above has written it).  Returns false when the wait ran out; clears
// range when the entry does not fit the window (lo to 32767 - near).
template <class A>
__device__ __forceinline__ bool commit2(const A &a, uint32_t *slot, int32_t strip, int32_t c, int4 h, int32_t base,
                                        int32_t lo, int32_t near, bool &range) {
    if (strip > 0 && (h.y != strip - 1 || h.w != strip - 1)) {
        const long long t0 = clock64();
        const long long limit = a.wait_limit > 0 ? a.wait_limit : kWaitLimitCycles;
        for (;;) {
            h = ld_ll(a.hbuf + c);
            if (h.y == strip - 1 && h.w == strip - 1) break;
            if (ld_volatile(&a.err[1]) != 0 || clock64() - t0 > limit) return false;
            __nanosleep(32);
        }
    }
    const int32_t d = h.z - base, ho = half16((uint32_t)h.x, 0) + d, f = half16((uint32_t)h.x, 1) + d;
    if (max(ho, f) > 32767 - near || min(ho, f) < lo) range = false;
    *slot = ((uint32_t)ho & 0xFFFFu) | ((uint32_t)f << 16);
    return true;
}

// What a column outside the matrix is read as: a mismatch for every row.
template <bool TAB>
__device__ __forceinline__ uint32_t no_column(int32_t mm1) {
    return TAB ? (uint32_t)(uint8_t)(int8_t)mm1 * 0x01010101u : 257u;
}

// Keeps column c's value.
__device__ __forceinline__ void put_col(uint32_t *col, int32_t c, uint32_t v) {
    const int32_t q = c & (kColRing - 1);
    col[q] = v;
    if (q < kRun) col[kColRing + q] = v;
}

// A strip that reaches past the rectangle's last row, after every lane has passed column
// 0 (step 64): its rows past the end, which went on from the left border (no cell of
// the rectangle, so the predicated steps before kept them out of the maxima), start
// again a gap below the lane's last row, or below a cell of the strip.  From here on
// they come from cells alone, a mismatch or a gap below them, and the steps need not
// tell them apart.
template <int RH>
__device__ __forceinline__ void drop_past_rows(Lane2<RH> &L, uint32_t rows, int64_t r_lane, int64_t m, uint32_t open2) {
    int32_t low = INT_MAX;  // the lowest H + open of the halves' first rows
    if (rows & 1u) low = half16(L.HO[0], 0);
    if (rows & 0x10000u) low = min(low, half16(L.HO[0], 1));
    const uint32_t low2 = dup16(__reduce_min_sync(0xffffffffu, low));
    uint32_t past = low2;
#pragma unroll
    for (int i = 0; i < RH; ++i) {
        const uint32_t in = ((rows >> i) & 0x00010001u) * 0xFFFFu;
        L.E[i] = (L.E[i] & in) | (past & ~in);
        L.HO[i] = (L.HO[i] & in) | (past & ~in);
        past = (__vadd2(L.HO[i], open2) & in) | (past & ~in);
    }
    // the row above the half is past the end too
    const uint32_t up = (r_lane <= m ? 0xFFFFu : 0u) | (r_lane + 32 * RH <= m ? 0xFFFF0000u : 0u);
    L.inHO = (L.inHO & up) | (low2 & ~up);
    L.inF = (L.inF & up) | (low2 & ~up);
    L.hod = (L.hod & up) | (low2 & ~up);
}

// The window of the bottom rows' offsets: the margin covers the rows above them
// and the columns until the next check (both neighbours' included).
struct Window2 {
    int32_t lo, hi;      // bottom-row offsets (H + open) allowed with base > 0; hi also with base = 0
    int32_t near;        // how far from both ends of the 16 bits an entry from outside has to be
    int32_t reach;       // no cell of the next run exceeds a lane's bottom row by more
};
template <int RH>
__device__ __forceinline__ Window2 window2(int32_t open, int32_t ext, int32_t mt1) {
    const int32_t e = min(-open, -ext), slope = mt1 + open + e;
    Window2 w;
    w.near = (RH + kRun) * slope - 2 * open;
    const int32_t margin = (RH + 2 * kRun) * slope - 4 * open + w.near + 64;
    w.lo = margin;
    w.hi = 32767 - margin;
    w.reach = kRun * slope + (RH - 1) * e - 2 * open;
    return w;
}

// Writes the rows of one half of a special column: HO and E of the lane's rows from
// its registers (lane 0, see run_strip2) or from shared memory.
template <int RH, class A>
__device__ __forceinline__ void put_special(const A &a, const Lane2<RH> &L, const WarpMem<RH> *w, int lane, int h,
                                            int32_t j, int64_t r_lane, int32_t base) {
    const int64_t r0 = r_lane + h * 32 * RH;
    int2 *dst = a.scols + (int64_t)((j + 1) / a.sc_every - 1) * a.m + r0;
    const bool pairs = RH % 2 == 0 && r0 + RH <= a.m && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
    for (int i = 0; i < RH; i += 2) {
        const int i1 = i + 1 < RH ? i + 1 : i;
        uint4 v = make_uint4(L.HO[i], L.HO[i1], L.E[i], L.E[i1]);
        if (lane > 0) v = w->spec[i / 2][lane];
        const int4 x = make_int4(half16(v.x, h) + base - a.open, half16(v.z, h) + base, half16(v.y, h) + base - a.open,
                                 half16(v.w, h) + base);
        if (pairs) {
            reinterpret_cast<int4 *>(dst)[i / 2] = x;
        } else {
            if (r0 + i < a.m) dst[i] = make_int2(x.x, x.y);
            if (i1 > i && r0 + i1 < a.m) dst[i1] = make_int2(x.z, x.w);
        }
    }
}

// The kRun steps from step k in a loop of SUB unrolled ones; the next step's inputs
// are loaded ahead.  spec: SC, the step after which my rows go to the special column.
// rows: ROWS, see step2.
template <int SUB, int RH, bool TAB, bool TRACK, int MODE, bool STORES, bool SC>
__device__ __forceinline__ void steps2(Lane2<RH> &L, const uint32_t *ra, const Consts2 &c, const uint32_t *pa,
                                       const uint32_t *pb, const uint32_t *rg, int4 *hb, int2 *st, uint4 (*sp)[32],
                                       int lane, Turn t, int spec, int32_t k, int32_t n, uint32_t rows, uint32_t &mx) {
    uint32_t ca = pa[0], cb = pb[0], rv = rg[0];
#pragma unroll 1
    for (int v = 0; v < kRun; v += SUB) {
        if (SC) t.spec = spec - v;
#pragma unroll
        for (int u = 0; u < SUB; ++u) {
            // the entry past the run's last is not used (it is inside the warp's memory)
            const uint32_t na = pa[v + u + 1], nb = pb[v + u + 1], nv = rg[v + u + 1];
            const uint32_t mask = MODE >= kPred ? active2(k + v + u, lane, n) : ~0u;
            const bool inside = MODE == kPlain || (uint32_t)(k + v + u - 63) < (uint32_t)n;
            step2<RH, TAB, TRACK, MODE, STORES, SC>(L, ra, c, ca, cb, rv, hb + v + u, st + v + u, sp, u, lane, t, inside,
                                                    mask, rows, mx);
            ca = na;
            cb = nb;
            rv = nv;
        }
    }
}

// What a launch may keep or be given besides the best cell: nothing; special rows and
// columns; a block's boundaries and wanted borders; a block with a left boundary whose
// last strip reaches past its last row.  Each has its own kernels: what they run
// between the runs of steps is bound by instruction fetch, and compiled into the
// pairs' kernels the blocks' code cost 2 to 6% (172 kbp pair 21.0 ms with all of it in,
// 20.5 with what it had of it before, 19.8 with none; 131 kbp block 12.6 ms with the
// last kind's code in, 12.3 without).
enum : int { kScore = 0, kStores = 1, kBorders = 2, kRagged = 3 };

// Runs strip s.  w->best_* holds the warp's best cell (kept over strips by the
// caller).
// Returns kErrNone, kErrTimeout or kErrRange.
template <int RH, bool TAB, int KIND, class A>
__device__ int32_t run_strip2(const A &a, WarpMem<RH> *w, int lane, int32_t s) {
    constexpr bool STORES = KIND != kScore, BORDERS = KIND >= kBorders, RAGGED = KIND == kRagged;
    // (the score-only kernels have no left boundary either; without its code the
    // compiler's schedule of their steps is worse: score only, 61 kbp 3.79 -> 3.89 ms)
    constexpr bool LEFT = BORDERS || KIND == kScore;
    Lane2<RH> L;
    uint32_t ra[RH];
    constexpr int64_t HR = 32 * RH;  // rows of a half
    const int64_t row0 = (int64_t)s * 2 * HR;
    const int64_t r_lane = row0 + (int64_t)lane * RH;  // my low half's first row
    const int32_t n = (int32_t)a.n;
    const Consts2 c = consts2(a.open, a.ext, a.gx, a.mt1, a.mm1);
    const Window2 win = window2<RH>(a.open, a.ext, a.mt1);

    Out2 o{{nullptr, nullptr}};
    if constexpr (STORES) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t q = 2 * (int64_t)s + h + 1;  // half strips above and including this one
            if (a.srows != nullptr && q % a.sr_every == 0 && q * HR <= a.m) o.row[h] = a.srows + (q / a.sr_every - 1) * a.n;
            if (BORDERS && a.bottom != nullptr && q * HR == a.m) o.row[h] = a.bottom;
        }
    }

    // left boundary: the base first, then offsets
    int32_t base = 0;
    if (LEFT && a.left) {
        int32_t lo = INT_MAX, hi = INT_MIN;
        for (int64_t i = lane; i < 2 * HR && row0 + i < a.m; i += 32) {
            const int2 lv = a.left[row0 + i];
            lo = min(lo, lv.x + a.open);
            hi = max(hi, max(lv.x + a.open, lv.y));
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lo / 2 + hi / 2 > 16384) base = lo / 2 + hi / 2 - 16384;
        if (hi - base > win.hi || (base > 0 && lo - base < win.lo)) return kErrRange;
    }
#pragma unroll
    for (int i = 0; i < RH; ++i) {
        uint32_t ho[2], ee[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            ho[h] = (uint32_t)a.open;  // H = 0 and E = 0 left of column 0
            ee[h] = 0u;
            if (LEFT && a.left) {
                // rows past the end repeat the last row's boundary
                const int64_t r = r_lane + h * HR + i;
                const int2 lv = a.left[r < a.m ? r : a.m - 1];
                ho[h] = (uint32_t)(lv.x + a.open - base);
                ee[h] = (uint32_t)max(lv.y - base, -16384);
            }
        }
        ra[i] = row2<RH, TAB>(a.rcode, a.rows, a.m, r_lane + i);
        L.HO[i] = (ho[0] & 0xFFFFu) | (ho[1] << 16);
        L.E[i] = (ee[0] & 0xFFFFu) | (ee[1] << 16);
    }
    int32_t corner = a.open;  // H + open above row 0 left of column 0
    if (BORDERS && s == 0) corner = a.corner + a.open - base;
    else if (BORDERS && a.left) corner = a.left[row0 - 1].x + a.open - base;
    if (corner > 32767 - win.near || corner < (base > 0 ? win.near : -32768)) return kErrRange;
    Turn t;
    t.selH = lane == 31 ? 0x5410u : 0x7654u;
    t.selF = lane == 31 ? 0x5432u : 0x7654u;
    t.hand = lane == 31 && row0 + 2 * HR < a.m && !(a.withhold && s == 0);
    t.keep = lane == 31 && (o.row[0] || o.row[1]);
    t.tag = s;
    t.base = base;

    // column 0's row above, then the first run's (columns 1..32) and column values
    // [0, 64).  From here on both are loaded a run before they are stored, more
    // than the ~800 cycles of an L2 round trip.
    int32_t wlo = base > 0 ? win.lo : -32768, wnear = base > 0 ? win.near : -32768;  // the window's lower ends
    {
        bool ok = true, range = true;
        if (lane == 0) ok = commit2(a, w->ring, s, 0, above2<BORDERS>(a, s, 0), base, wnear, win.near, range);
        if (!__all_sync(0xffffffffu, ok && range)) return __all_sync(0xffffffffu, ok) ? kErrRange : kErrTimeout;
    }
    __syncwarp();
    {
        // what the shuffles of the step before column 0 would have brought
        const uint32_t up = __shfl_sync(0xffffffffu, L.HO[RH - 1], (lane + 31) & 31);
        const uint32_t v = w->ring[0];
        L.hod = lane == 0 ? ((uint32_t)corner & 0xFFFFu) | (up << 16) : up;
        L.inHO = lane == 0 ? (v & 0xFFFFu) | (up << 16) : up;
        const uint32_t zero = dup16(a.gx);  // F below H = 0
        L.inF = lane == 0 ? (v >> 16) | (zero & 0xFFFF0000u) : zero;
    }
    __syncwarp();
    int4 up4 = make_int4(0, 0, 0, 0);
    if (1 + lane < n) up4 = above2<BORDERS>(a, s, 1 + lane);
    // Columns outside the matrix mismatch every row.  Left of it (no left boundary
    // given) H then stays 0 and the steps need no predicate; E is open there where
    // the recurrence starts from 0, which is gone after |open| / |extend| columns and
    // never positive.  Right of it the values belong to no cell and reach none: they
    // stay below a cell's value that was seen before, and the exact rerun, the
    // stored rows and the special columns leave them out.  A given boundary (they
    // would go on from it, and it is no cell) or a wanted right border needs the
    // predicates.
    const bool exact = BORDERS && (a.top != nullptr || a.left != nullptr || a.right != nullptr);
    const uint32_t none = no_column<TAB>(a.mm1);
    put_col(w->col, lane, col_value<TAB>(lane < n ? read_col<TAB>(a.ctab, a.cols, lane) : none));
    put_col(w->col, lane - 32, col_value<TAB>(none));
    put_col(w->col, lane - 64, col_value<TAB>(none));
    uint32_t cv = kRun + lane < n ? read_col<TAB>(a.ctab, a.cols, kRun + lane) : none;
    if (a.trace && lane == 0) {  // the strip above has delivered column 0
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        a.trace[3 * s] = (int64_t)now;
    }

    const bool past_end = RAGGED && row0 + 2 * HR > a.m;
    const uint32_t rows_here = RAGGED ? rows_in<RH>(r_lane, a.m) : 0u;

    // the best H known anywhere, loaded a run before it is used
    int32_t gpre = ld_volatile(a.gbest);
    int32_t thr = max(w->best_ho, gpre + a.open);
    // kept runs: slots first, first + 1, ... (cyclic), all with maximum kv
    int first = 0, kept = 0;
    int32_t kv = 0;
    const int32_t kEnd = n + 63;
    for (int32_t k = 0;; k += kRun) {
        const bool end = k >= kEnd;
        if (end || kept == kKept<RH>) {
            // the kept runs again, unless a better cell was found elsewhere; in the
            // middle of the strip the lanes' rows wait in shared memory
            if constexpr (BORDERS) {
                if (end && a.right != nullptr) {
                    // after its last column a half's registers hold H + open and E of column n - 1
#pragma unroll
                    for (int i = 0; i < RH; ++i)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int64_t r = r_lane + h * HR + i;
                            if (r < a.m) a.right[r] = make_int2(half16(L.HO[i], h) + base - a.open, half16(L.E[i], h) + base);
                        }
                }
            }
            const uint32_t inHO = L.inHO, inF = L.inF, hod = L.hod;
            if (!end) {
#pragma unroll
                for (int i = 0; i < RH; i += 2) {
                    const int i1 = i + 1 < RH ? i + 1 : i;
                    w->spec[i / 2][lane] = make_uint4(L.HO[i], L.HO[i1], L.E[i], L.E[i1]);
                }
            }
            if (kv >= __shfl_sync(0xffffffffu, ld_volatile(a.gbest), 0) + a.open) {
#pragma unroll 1
                for (int q = 0; q < kept; ++q)
                    rerun<RH, TAB, RAGGED>(a, w, L, ra, c, first + q < kKept<RH> ? first + q : first + q - kKept<RH>, lane, r_lane);
            }
            kept = 0;
            if (end) break;
#pragma unroll
            for (int i = 0; i < RH; i += 2) {
                const int i1 = i + 1 < RH ? i + 1 : i;
                const uint4 v = w->spec[i / 2][lane];
                L.HO[i] = v.x;
                L.E[i] = v.z;
                L.HO[i1] = v.y;
                L.E[i1] = v.w;
            }
            L.inHO = inHO;
            L.inF = inF;
            L.hod = hod;
        }
        if (past_end && k == 64) drop_past_rows(L, rows_here, r_lane, a.m, c.open2);
        // refill: the next run's row above and the columns of the run after it in.  One
        // vote says whether every lane is inside its window and every entry is there
        // and close to the base; the lanes that would wait or move the base are rare.
        const uint32_t bot = L.HO[RH - 1];
        const int32_t vmax = max16(bot), vmin = min(half16(bot, 0), half16(bot, 1));
        const int32_t q = k + 1 + lane, qc = k + kRun + lane;
        const int32_t ub = up4.z - base, uho = half16((uint32_t)up4.x, 0) + ub, uf = half16((uint32_t)up4.x, 1) + ub;
        thr = max(thr, gpre + a.open);
        bool near = vmax + win.reach >= thr - base;  // some cell of this run may reach the best known
        if (BORDERS && a.top != nullptr) {
            // a given top border may rise from column to column as no matrix does, and
            // with it the strips' rows above: what they bring into this run counts too
            // (the entries not there yet: below)
            const int32_t up = max16(__vimax3_s16x2(L.inHO, L.hod, L.inF));
            near |= max(up, q < n ? max(uho, uf) : up) + win.reach >= thr - base;
        }
        bool track = __any_sync(0xffffffffu, near);
        const bool mine = vmax <= win.hi && vmin >= wlo;
        const bool entry = q >= n || (max(uho, uf) <= 32767 - win.near && min(uho, uf) >= wnear &&
                                      (s == 0 || (up4.y == s - 1 && up4.w == s - 1)));
        if (__all_sync(0xffffffffu, mine && entry)) {
            w->ring[lane] = q < n ? ((uint32_t)uho & 0xFFFFu) | ((uint32_t)uf << 16) : bot;  // past the end any value of the window
        } else {
            if (__any_sync(0xffffffffu, !mine)) {
                // the base moves so that the bottom rows are in the middle of the window
                const int32_t hi = __reduce_max_sync(0xffffffffu, vmax), lo = __reduce_min_sync(0xffffffffu, vmin);
                const int32_t mid = base + (lo + hi) / 2;
                const int32_t nb = mid > 16384 ? mid - 16384 : 0;
                const int32_t d = base - nb;
                if (hi + d > win.hi || (nb > 0 && lo + d < win.lo)) return kErrRange;
                const uint32_t d2 = dup16(d);
#pragma unroll
                for (int i = 0; i < RH; ++i) {
                    L.HO[i] = __vadd2(L.HO[i], d2);
                    L.E[i] = __vadd2(L.E[i], d2);
                }
                L.inHO = __vadd2(L.inHO, d2);
                L.inF = __vadd2(L.inF, d2);
                L.hod = __vadd2(L.hod, d2);
                base = nb;
                t.base = base;
                wlo = base > 0 ? win.lo : -32768;
                wnear = base > 0 ? win.near : -32768;
            }
            bool ok = true, range = true;
            if (q < n) ok = commit2(a, w->ring + lane, s, q, up4, base, wnear, win.near, range);
            else w->ring[lane] = L.HO[RH - 1];
            if (!__all_sync(0xffffffffu, ok && range)) return __all_sync(0xffffffffu, ok) ? kErrRange : kErrTimeout;
            if (BORDERS && a.top != nullptr) {
                track |= __any_sync(0xffffffffu, max16(w->ring[lane]) + win.reach >= thr - base);
            }
        }
        put_col(w->col, qc, col_value<TAB>(cv));
        if (s > 0) {
            ld_hand(up4, q + kRun < n, a.hbuf + (q + kRun));
        } else if (BORDERS && a.top && q + kRun < n) {
            up4 = above2<BORDERS>(a, s, q + kRun);
        }
        cv = none;
        ld_col<TAB>(cv, qc + kRun < n, a.ctab, a.cols, qc + kRun);
        ld_best(gpre, a.gbest);
        const int32_t rel = thr - base;
        __syncwarp();

        const uint32_t *pa = w->col + ((k - lane) & (kColRing - 1)), *pb = w->col + ((k - lane - 32) & (kColRing - 1));
        int4 *hb = a.hbuf + ((int64_t)k - 63);
        // a special column j (j + 1 a multiple of sc_every, itself one of 128) meets
        // lane l's low half at step j + l and its high half 32 steps later: steps 1 to
        // 31 of the run at k = j + 1 and of the next one, and for lane 0 the step
        // before each, so that its registers hold the column when the run begins
        const bool sc_run = STORES && a.scols != nullptr && (k & (a.sc_every - 1)) <= 32 && k >= a.sc_every;
        const int mode = k >= 64 && k + kRun <= n ? kPlain : (exact ? kPred : kEdge);
        uint32_t mx = 0x80008000u;
        const int cur = first + kept < kKept<RH> ? first + kept : first + kept - kKept<RH>;
        if (!track && mode == kPlain && !sc_run) {
            steps2<Sub<RH>::plain, RH, TAB, false, kPlain, STORES, false>(L, ra, c, pa, pb, w->ring, hb, w->stage, w->spec, lane, t,
                                                                 -1, k, n, rows_here, mx);
        } else {
            if (sc_run && lane == 0) {
                const int h = (k & (a.sc_every - 1)) == 0 ? 0 : 1;
                if (k - 1 - 32 * h < n) put_special(a, L, w, 0, h, k - 1 - 32 * h, r_lane, base);
            }
            put_state(w, cur, lane, L);
            w->sring[cur][lane] = w->ring[lane];
            const int spec = sc_run ? lane - 1 : -1;
            if (mode == kPlain && !sc_run)
                steps2<Sub<RH>::plain, RH, TAB, true, kPlain, STORES, false>(L, ra, c, pa, pb, w->ring, hb, w->stage, w->spec, lane,
                                                                    t, -1, k, n, rows_here, mx);
            else if (STORES && mode == kPlain)
                steps2<Sub<RH>::edge, RH, TAB, true, kPlain, STORES, STORES>(L, ra, c, pa, pb, w->ring, hb, w->stage, w->spec, lane,
                                                                      t, spec, k, n, rows_here, mx);
            else if (!BORDERS || mode == kEdge)
                steps2<Sub<RH>::edge, RH, TAB, true, kEdge, STORES, STORES>(L, ra, c, pa, pb, w->ring, hb, w->stage, w->spec, lane,
                                                                       t, spec, k, n, rows_here, mx);
            else if (RAGGED && past_end)
                steps2<1, RH, TAB, true, kPredRows, STORES, STORES>(L, ra, c, pa, pb, w->ring, hb, w->stage, w->spec, lane,
                                                                       t, spec, k, n, rows_here, mx);
            else
                steps2<1, RH, TAB, true, kPred, STORES, STORES>(L, ra, c, pa, pb, w->ring, hb, w->stage, w->spec, lane,
                                                                       t, spec, k, n, rows_here, mx);
        }
        // the run's stored rows and special column out
        if constexpr (STORES) {
            __syncwarp();
            if (o.row[0] || o.row[1]) flush2(w, lane, o, n, k + kRun, base, a.open);
            if (sc_run && lane > 0) {
                const int h = (k & (a.sc_every - 1)) == 0 ? 0 : 1;
                if (k - 1 - 32 * h < n) put_special(a, L, w, lane, h, k - 1 - 32 * h, r_lane, base);
            }
        }
        // did it reach the best H known?
        const int32_t top = max16(mx);
        if ((track || mode != kPlain || sc_run) && __any_sync(0xffffffffu, top >= rel)) {
            const int32_t val = __reduce_max_sync(0xffffffffu, top) + base;
            if (lane == 0) {
                if (val > thr) atomicMax(a.gbest, val - a.open);
                w->kept_k[cur] = k;
                w->kept_base[cur] = base;
                w->kept_val[cur] = val;
            }
            thr = val;
            if (kept > 0 && kv == val) {
                ++kept;
            } else {
                first = cur;
                kept = 1;
                kv = val;
            }
        }
    }
    __syncwarp();
    return kErrNone;
}

}  // namespace
}  // namespace swb

// warp.cuh - one banded POA alignment by one warp: the value fill of team.cuh
// (same cells, same arithmetic, same backtrack) for the batch kernel, where
// thousands of windows run at once and the instructions per cell are the cost.
//
// A lane owns a block of 8 cells; chunk c of a row is blocks Bs + 32 c .. of
// it, so a row of a 500 bp window (29-31 blocks) is one chunk with no idle
// strip ends, and the left neighbour of a block is the previous lane's. Rows
// go to the slot's row store, 32 bytes per block; with the static band the
// last rows are also kept in a shared-memory ring (two planes of 16 bytes per
// block, so any shift between a row's band and its predecessor's reads without
// bank conflicts). With the dynamic bands the ring is a circular buffer of blocks
// that holds as many of the last rows as fit, whatever their width.
//
// Measured on a B200 against the record fill it replaced (kernel time, with the
// graph steps of batch.cu): 8,000 polishing windows 651 -> 207 ms, 1,024 windows of
// 2,000 bp at 15 % error with the adaptive band 1,118 -> 349 ms, one window of 64
// reads 282 -> 94 ms. What is left is latency: of 3.9 cycles an instruction of a
// lone warp (adaptive band) 1.5 wait for an earlier instruction, 0.65 for global and
// 0.36 for shared memory; static band 4.9, 1.8, 1.05 and 0.63.
#pragma once
#include "team.cuh"

namespace pb {

constexpr int WSTG = 16, WSTG_E = 64;  // rows and predecessor records staged at a time (static band)
constexpr int WSTG_BYTES = WSTG * 16 + WSTG_E * 16;
constexpr int WED = 32;                // an adaptive row's predecessor records in shared memory
// shared memory of the adaptive fill: records, then the state window
constexpr int warp_state_bytes(int rows) { return rows * SW_INTS * 4; }

// Shared-memory copies of rows. A row's blocks lie between two blocks of
// unreachable cells, so a lane outside a predecessor's band reads those instead
// of taking another path.
struct WarpRing {
    unsigned at;  // shared memory address
    int rows;     // static band: a power of two, or 0: no ring
    int blocks;   // static band: blocks per row
    int cur;      // dynamic bands: the current row's first block (of its pads), or -1: not kept
};
enum { RING_STATIC = 1, RING_DYN = 2 };
constexpr int warp_ring_row_blocks(int blocks) { return blocks + 2; }

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
    return d;
}
// byte l of x, sign-extended
template <int l>
__device__ __forceinline__ int32_t sbyte(uint32_t x) { return (int32_t)prmt(x, x, 0x8880u + 0x1111u * l); }

// The query for the warp fill: codes as nibbles, eight columns a word.
// qcode: the code of one column.
__device__ __forceinline__ int qcode(const uint32_t* qn, int col) { return (int)(qn[col >> 3] >> (4 * (col & 7))) & 15; }

// a record's base as warp_row takes it
template <bool WIDE>
__device__ __forceinline__ int row_score(const CellK& k, int base) { return WIDE ? base : (int)score_table(k, base); }

// One row. ed_at(e): {ring offset, or ~row-store block; base (WIDE) or score
// table; Bs; last block - Bs}. With ARGMAX, best / best_col become the row's first maximum.
// U chunks are taken together: a chunk is ~300 mostly dependent instructions, so
// two of them in flight hide each other's latency where the registers allow it
// (rows of several chunks, few warps per SM).
//
// The query codes are byte selectors: one PRMT turns a predecessor's score table
// into the scores of four cells.
//
// The gap term of cell l is I[l] = max(I[l-1] + e1, H0[l-1] + o1): within a
// block one dependent step per cell, first from nothing for the block's own
// contribution, then from the prefix over the lanes.
template <bool WIDE, int RING, bool ARGMAX, int U, class EdAt>
__device__ __forceinline__ void warp_row(const CellK& k, int i, int Bs, int span, int tb, int d, const uint32_t* qn,
                                         const WarpRing& ring, char* store, int lane, EdAt ed_at, int32_t& best,
                                         int& best_col) {
    typedef Cells<WIDE> C;
    constexpr int32_t NEG = C::NEG;
    constexpr int32_t LOW = WIDE ? INT_MIN : -(1 << 30);
    constexpr int HB = 4 * C::BYTES, BB = 2 * HB;  // bytes per half block and block
    // gap terms are kept as their value at column 0 (minus j * e1); the floor: NEG_INF extended from column 0
    int32_t carry = NEG;
    // row 0 has no gap terms: they start, and open, below everything
    constexpr int32_t BELOW = WIDE ? -2000000000 : -(1 << 30);
    const int32_t open = i == 0 && !WIDE ? BELOW : k.o1;
    for (int c0 = 0; c0 <= span; c0 += 32 * U) {
        int32_t H[U][8], V[U][8], out[U];
        uint32_t qw[U];
        bool act[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int b = c0 + 32 * u + lane;
            act[u] = b <= span;
            qw[u] = qn[Bs + min(b, span)];
#pragma unroll
            for (int l = 0; l < 8; l++) { H[u][l] = NEG; V[u][l] = NEG - k.o1; }
            if (i == 0 && Bs + b == 0) H[u][0] = 0;
        }
        for (int e = 0; e < d; e++) {
            const int4 er = ed_at(e);
            C lo[U], hi[U];
            int32_t left0[U];  // lane 0: the cell before the chunk (NEG_INF before the row's first block)
            bool in[U];
            if (er.x >= 0) {
                const int plane = (RING == RING_STATIC ? ring.blocks + 2 : er.w + 3) * HB;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int pb = Bs + c0 + 32 * u + lane - er.z;
                    in[u] = (unsigned)pb <= (unsigned)er.w;
                    const unsigned src = ring.at + er.x + (min(max(pb, -1), er.w + 1) + 1) * HB;
                    lo[u].lds(src);
                    hi[u].lds(src + plane);
                    left0[u] = NEG;
                    if (c0 + u > 0) left0[u] = C::lds_m(ring.at + er.x + plane + (min(max(pb - 1, -1), er.w + 1) + 1) * HB + HB - C::BYTES);
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int pb = Bs + c0 + 32 * u + lane - er.z;
                    in[u] = act[u] && (unsigned)pb <= (unsigned)er.w;
                    const char* src = store + ((int64_t)~er.x + pb) * BB;
                    left0[u] = NEG;
                    if (in[u]) { lo[u].load(src); hi[u].load(src + HB); }
                    else { lo[u].none(); hi[u].none(); }
                    if (lane == 0 && c0 + u > 0 && in[u] && pb > 0) left0[u] = C::load_m(src - C::BYTES);
                }
            }
            const uint32_t tabn = WIDE ? 0u : (uint32_t)(er.y == (int)score_table(k, 4) ? k.match : k.mismatch);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int B = Bs + c0 + 32 * u + lane;
                // the fill's block mask for the diagonal (src/align.cpp:1467)
                const bool diag = in[u] && (B > er.z || B == 0);
                int32_t left = __shfl_up_sync(0xffffffffu, hi[u].m(3), 1);
                if (lane == 0) left = left0[u];
                if (diag) {
                    if constexpr (WIDE) {
#pragma unroll
                        for (int l = 0; l < 8; l++) {
                            const int32_t src = l == 0 ? left : l <= 4 ? lo[u].m(l > 0 ? l - 1 : 0) : hi[u].m(l - 5);
                            H[u][l] = mx(H[u][l], src + ((int)((qw[u] >> (4 * l)) & 15u) == er.y ? k.match : k.mismatch));
                        }
                    } else {
                        const uint32_t s0 = prmt((uint32_t)er.y, tabn, qw[u]), s1 = prmt((uint32_t)er.y, tabn, qw[u] >> 16);
                        H[u][0] = mx(H[u][0], left + sbyte<0>(s0));
                        H[u][1] = mx(H[u][1], lo[u].m(0) + sbyte<1>(s0));
                        H[u][2] = mx(H[u][2], lo[u].m(1) + sbyte<2>(s0));
                        H[u][3] = mx(H[u][3], lo[u].m(2) + sbyte<3>(s0));
                        H[u][4] = mx(H[u][4], lo[u].m(3) + sbyte<0>(s1));
                        H[u][5] = mx(H[u][5], hi[u].m(0) + sbyte<1>(s1));
                        H[u][6] = mx(H[u][6], hi[u].m(1) + sbyte<2>(s1));
                        H[u][7] = mx(H[u][7], hi[u].m(2) + sbyte<3>(s1));
                    }
                }
#pragma unroll
                for (int l = 0; l < 8; l++) V[u][l] = mx(V[u][l], l < 4 ? lo[u].v(l & 3, k) : hi[u].v(l & 3, k));
            }
        }
        // H0; what the block passes on by itself; the row's maximum
#pragma unroll
        for (int u = 0; u < U; u++) {
#pragma unroll
            for (int l = 0; l < 8; l++) H[u][l] = mx(H[u][l], add32(V[u][l], k.o1));
            int32_t t = add32(H[u][0], open);
#pragma unroll
            for (int l = 1; l < 8; l++) t = mx(add32(t, k.e1), add32(H[u][l], open));
            out[u] = act[u] ? t - ((c0 + 32 * u + lane + 1) * BLK) * k.e1 : LOW;
            if (ARGMAX) {
                // the first maximum of H0 is the row's first maximum (a gap never exceeds the cell it opens from)
                const int32_t lm = act[u] ? mx(mx(mx(H[u][0], H[u][1]), mx(H[u][2], H[u][3])),
                                               mx(mx(H[u][4], H[u][5]), mx(H[u][6], H[u][7]))) : INT_MIN;
                const int32_t wm = __reduce_max_sync(0xffffffffu, lm);
                if (wm > best) {
                    best = wm;
                    int l = 7;
#pragma unroll
                    for (int q = 6; q >= 0; q--) l = H[u][q] == wm ? q : l;
                    best_col = __shfl_sync(0xffffffffu, (Bs + c0 + 32 * u + lane) * BLK + l,
                                           __ffs(__ballot_sync(0xffffffffu, lm == wm)) - 1);
                }
            }
        }
        int32_t incl[U];
#pragma unroll
        for (int u = 0; u < U; u++) incl[u] = scan_max(out[u]);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int b = c0 + 32 * u + lane;
            int32_t ex = __shfl_up_sync(0xffffffffu, incl[u], 1);
            if (lane == 0) ex = LOW;
            int32_t I = mx(carry, ex) + (b * BLK) * k.e1;
            carry = mx(carry, __shfl_sync(0xffffffffu, incl[u], 31));
            if (i == 0) I = BELOW;
            C lo, hi;
#pragma unroll
            for (int l = 0; l < 8; l++) {
                const int32_t h = H[u][l], M = mx(h, I);
                if (l < 4) lo.set(l & 3, M, V[u][l], k);
                else hi.set(l & 3, M, V[u][l], k);
                I = mx(add32(I, k.e1), WIDE && i == 0 ? BELOW : add32(h, open));
            }
            if (act[u]) {
                if (RING == RING_STATIC ? span < ring.blocks : ring.cur >= 0) {
                    const unsigned at = RING == RING_STATIC ? (i & (ring.rows - 1)) * (unsigned)((ring.blocks + 2) * BB) : ring.cur * BB;
                    const unsigned dst = ring.at + at + (b + 1) * HB, plane = (RING == RING_STATIC ? ring.blocks + 2 : span + 3) * HB;
                    lo.sts(dst);
                    hi.sts(dst + plane);
                    if (b == span) {
                        C pad;
                        pad.none();
                        pad.sts(dst + HB);
                        pad.sts(dst + plane + HB);
                    }
                    if (RING == RING_DYN && b == 0) {  // (the static ring's are written once)
                        C pad;
                        pad.none();
                        pad.sts(dst - HB);
                        pad.sts(dst + plane - HB);
                    }
                }
                char* dst = store + ((int64_t)tb + b) * BB;
                lo.store(dst);
                hi.store(dst + HB);
            }
        }
    }
}

// Static band: rows and records staged WSTG rows at a time.
template <bool WIDE>
__device__ void warp_fill_static(const TeamJob& a, const WarpRing& ring, const uint32_t* qsm, unsigned char* stage, int lane) {
    const int n = a.n;
    const CellK k = a.k;
    char* const store = a.store;
    const unsigned stg = (unsigned)__cvta_generic_to_shared(stage);
    int32_t bm = 0;
    int bc = 0;
    {
        // the blocks before the ring's rows
        constexpr int HB = 4 * Cells<WIDE>::BYTES;
        Cells<WIDE> pad;
        pad.none();
        for (int x = lane; x < 2 * ring.rows; x += 32) pad.sts(ring.at + x * (ring.blocks + 2) * HB);
    }
    for (int i0 = 0; i0 < n; i0 += WSTG) {
        const int cnt = min(WSTG, n - i0);
        const int e0 = a.in_ptr[i0], ne = min(a.in_ptr[i0 + cnt] - e0, WSTG_E);
        __syncwarp();
        if (lane < cnt) cp_async16(stage + lane * 16, a.fr + i0 + lane);
        for (int e = lane; e < ne; e += 32) cp_async16(stage + WSTG * 16 + e * 16, a.fe + e0 + e);
        cp_async_commit_all();
        cp_async_wait_all();
        __syncwarp();
        for (int x = 0; x < cnt; x++) {
            const int4 h = lds128(stg + x * 16);
            const unsigned ed = stg + WSTG * 16 + (h.w >> FR_EOFF) * 16;
            const int i = i0 + x;
            const int4* fe = a.fe;
            if (h.w & FR_UNSTAGED)
                warp_row<WIDE, RING_STATIC, false, 1>(k, i, h.x, h.y, h.z, h.w & FR_D, qsm, ring, store, lane,
                                                   [&](int e) { return fe[a.in_ptr[i] + e]; }, bm, bc);
            else
                warp_row<WIDE, RING_STATIC, false, 1>(k, i, h.x, h.y, h.z, h.w & FR_D, qsm, ring, store, lane,
                                                   [&](int e) { return lds128(ed + e * 16); }, bm, bc);
            __syncwarp();
        }
    }
}

// Adaptive band (-B) or full band (f = 0): bands known row by row. The band
// state's serial part is team_state's and team_records', on the same warp: inputs
// that do not need row i's maximum are fetched before the row is filled, the state
// of nearby rows lives in a shared-memory window of `wrows` rows (a power of two),
// their cells in a buffer of rcap blocks at `rbuf`. Returns a status (uniform).
//
// Of a 1,130-cell row's 9,300 cycles the serial part took 3,040: a wait for the
// state entering the window (500), lists in loops around a divergent branch (780
// for the records, 213 as one pass that reads the window whatever the row), and
// the state a word at a time. Now 1,540 (1,024 windows of 2,000 bp: 398 -> 365 ms).
template <bool WIDE, int U>
__device__ int warp_fill_dyn(const TeamJob& a, bool adaptive, unsigned char* wsm, int wrows, unsigned char* rbuf, int rcap,
                             const uint32_t* qf, int lane, int64_t& cells_out) {
    const int n = a.n, m = a.qlen + 1, E = a.in_ptr[n];
    const CellK k = a.k;
    char* const store = a.store;
    const unsigned seda = (unsigned)__cvta_generic_to_shared(wsm);
    int32_t* win = reinterpret_cast<int32_t*>(wsm + WED * 16);
    const int wmask = wrows - 1, AHEAD = wrows / 2 - 1;
    const unsigned wina = seda + WED * 16;
    // row r's state: {Pl, Pr, Ol, Or}, {Ow, Sl, Mp, rpos}, {Bs, Be, tb, rat}
    auto slot = [&](int r) { return wina + (r & wmask) * (SW_INTS * 4); };
    if (adaptive)
        for (int64_t x = lane; x < 8 * (int64_t)n; x += 32) a.state[x] = (x & 7) == SW_PL ? m : 0;
    for (int x = lane; x < wrows * SW_INTS; x += 32) win[x] = x % SW_INTS == SW_PL ? m : 0;
    __syncwarp();
    int4 ra0 = a.ra[0], ra1 = a.ra[1];            // row i
    int4 rb0 = make_int4(0, 0, 0, 0), rb1 = rb0;  // row i + 1
    if (n > 1) { rb0 = a.ra[2]; rb1 = a.ra[3]; }
    int Bs, Be;
    if (adaptive) band_adaptive(ra0.z, ra0.w, m, a.w, m, 0, 0, 0, 0, Bs, Be);
    else band_static(0, 0, 0, m, a.w, Bs, Be);
    Bs = 0;
    int64_t tb = 0, cells = 0;
    int edx = 0, edx_n = 0, succ = -1, succ_n = -1;
    int4 far = make_int4(0, 0, 0, 0);  // the row's predecessors beyond the window, one per lane: row,
    int2 far_s = make_int2(0, 0);      // slope and maximum
    if (lane < ra1.w) succ = a.out_row[ra0.y + lane];
    if (n > 1) {
        if (lane < rb1.z) edx_n = a.ed[rb0.x + lane].x;
        if (lane < rb1.w) succ_n = a.out_row[rb0.y + lane];
    }
    constexpr int BB = BLK * Cells<WIDE>::BYTES;
    WarpRing ring{(unsigned)__cvta_generic_to_shared(rbuf), 0, 0, -1};
    int rpos = 0, rat = 0;  // end of the stream of kept blocks; its place in the buffer
    for (int i = 0; i < n; i++) {
        const int bn = Be - Bs - 1;
        const int d = i == 0 ? 0 : ra1.z, ns = ra1.w;
        if (bn < 0) return ST_DEGENERATE;
        if (d > MAX_MULTI_PRED) return ST_INDEGREE;
        if (tb + bn > a.store_cap || tb + bn > INT_MAX) return ST_OOM;
        int4 rc0 = rb0, rc1 = rb1;
        int edx_2 = 0, succ_2 = -1;
        if (i + 2 < n) {
            rc0 = a.ra[2 * (i + 2)];
            rc1 = a.ra[2 * (i + 2) + 1];
            // (the in-window in-edges and out-edges are the same edges: E of each)
            const int e2 = rb0.x + rb1.z, o2 = rb0.y + rb1.w;
            if (e2 + lane < E) edx_2 = a.ed[e2 + lane].x;
            if (o2 + lane < E) succ_2 = a.out_row[o2 + lane];
        }
        int32_t pend = 0;  // state entering the window, one int per lane (8)
        if (adaptive && i >= 1 && i - 1 + AHEAD < n && lane < 8) pend = a.state[8 * (int64_t)(i - 1 + AHEAD) + lane];
        // the next row's predecessors beyond the window, whose rows are done
        int4 far_n = make_int4(0, 0, 0, 0);
        int2 far_sn = make_int2(0, 0);
        if (lane < rb1.z && i + 1 - (edx_n >> 4) >= AHEAD) {
            far_n = a.rowi[edx_n >> 4];
            if (adaptive) {
                const int32_t* w = a.state + 8 * (int64_t)(edx_n >> 4);
                far_sn = make_int2(w[SW_SL], w[SW_MP]);
            }
        }
        // the row's place in the buffer: whole, so the end of the buffer may stay empty
        ring.cur = -1;
        if (bn > 0 && bn + 2 <= rcap) {
            if (rat + bn + 2 > rcap) { rpos += rcap - rat; rat = 0; }
            ring.cur = rat;
            rat += bn + 2;
            rpos += bn + 2;
        }
        if (lane == 0) {
            a.rowi[i] = make_int4(Bs, Be, (int)tb, 0);
            sts128(slot(i) + 32, make_int4(Bs, Be, (int)tb, ring.cur));
            sts32(slot(i) + 28, rpos - bn - 2);
        }
        // row i's predecessor records; their slopes and maxima
        int psl = 0, pmp = INT_MIN / 2;
        auto put_record = [&](int kk, int x, int4 q, int from) {  // q: {Bs, Be, tb}; from: its first block in the buffer, or -1
            const int2 band = rec_band(q.x, q.y);
            if (kk < WED) sts128(seda + kk * 16, make_int4(from >= 0 ? from * BB : ~q.z, row_score<WIDE>(k, x & 7), band.x, band.y));
            a.ed[ra0.x + kk] = make_int4(x, q.x, q.y, q.z);
        };
        if (lane < d) {
            const int p = edx >> 4;
            const bool near = i - p < AHEAD;
            const int4 w = lds128(slot(p) + 16), q = lds128(slot(p) + 32);
            psl = near ? w.y : far_s.x;
            pmp = near ? w.z : far_s.y;
            // (written over in the buffer by now?)
            put_record(lane, edx, near ? q : far, near && rpos - w.w <= rcap ? q.w : -1);
        }
        for (int kk = 32 + lane; kk < d; kk += 32) {
            const int x = a.ed[ra0.x + kk].x;
            put_record(kk, x, a.rowi[x >> 4], -1);
        }
        __syncwarp();
        const int4 own0 = lds128(slot(i)), own1 = lds128(slot(i) + 16), nw = lds128(slot(i + 1));
        int sl = own1.y, ow = own1.x, ol = own0.z, orr = own0.w;
        int nPl = nw.x, nPr = nw.y, nOl = nw.z, nOr = nw.w, nOw = lds32(slot(i + 1) + 16);
        const int max_psl = adaptive ? __reduce_max_sync(0xffffffffu, psl) : 0;
        const int4* ed = a.ed + ra0.x;
        auto ed_at = [&](int e) {
            if (e < WED) return lds128(seda + e * 16);
            const int4 v = ed[e];
            const int2 band = rec_band(v.y, v.z);
            return make_int4(~v.w, row_score<WIDE>(k, v.x & 7), band.x, band.y);
        };
        int32_t best = INT_MIN;
        int acj = Bs * BLK;
        if (U > 1 && adaptive && bn > 32)
            warp_row<WIDE, RING_DYN, true, U>(k, i, Bs, bn - 1, (int)tb, d, qf, ring, store, lane, ed_at, best, acj);
        else if (adaptive)
            warp_row<WIDE, RING_DYN, true, 1>(k, i, Bs, bn - 1, (int)tb, d, qf, ring, store, lane, ed_at, best, acj);
        else
            warp_row<WIDE, RING_DYN, false, 1>(k, i, Bs, bn - 1, (int)tb, d, qf, ring, store, lane, ed_at, best, acj);
        cells += (int64_t)bn * BLK;
        tb += bn;
        if (adaptive) {
            if (i >= 1) {  // src/align.cpp:1516-1568
                // the state that enters the window (asked for before the row was filled)
                if (i - 1 + AHEAD < n && lane < 8) sts32(slot(i - 1 + AHEAD) + 4 * lane, pend);
                __syncwarp();
                int sl_best = INT_MIN, max_slp = 0;
                bool is_match = false;
                if (ra1.y == qcode(qf, acj + 1)) {  // cur.base == seq[max_acj]
                    max_slp = max_psl;
                    sl_best = __reduce_max_sync(0xffffffffu, pmp + 1 == acj ? psl + 1 : INT_MIN);
                    if (d > 32) {
                        for (int kk = 32 + lane; kk < d; kk += 32) {
                            const int p = ed[kk].x >> 4;
                            const int4 w = i - p < AHEAD ? lds128(slot(p) + 16)
                                                         : *reinterpret_cast<const int4*>(a.state + 8 * (int64_t)p + 4);
                            max_slp = max(max_slp, w.y);
                            if (w.z + 1 == acj) sl_best = max(sl_best, w.y + 1);
                        }
                        max_slp = __reduce_max_sync(0xffffffffu, max_slp);
                        sl_best = __reduce_max_sync(0xffffffffu, sl_best);
                    }
                    is_match = sl_best != INT_MIN;
                }
                if (is_match) sl = mx(sl, sl_best);
                if (!is_match && max_slp < 30) ow = mn(ow + max_slp + 1, 5 * a.w);
                if (sl >= 30) {
                    ol = orr = acj - ra1.x;
                    ow = 0;
                }
                auto put_state = [&](int sr) {
                    const bool near = sr - i < AHEAD;
                    int32_t* gs = a.state + 8 * (int64_t)sr;
                    int4 w = lds128(slot(sr));
                    int sow = lds32(slot(sr) + 16);
                    if (!near) {
                        w = *reinterpret_cast<const int4*>(gs);
                        sow = gs[SW_OW];
                    }
                    w = make_int4(mn(w.x, acj), mx(w.y, acj + 1), sl >= 30 ? ol : mn(w.z, ol), sl >= 30 ? orr : mx(w.w, orr));
                    sow = ow ? mx(sow, ow) : ow;
                    if (near) {
                        sts128(slot(sr), w);
                        sts32(slot(sr) + 16, sow);
                    } else {
                        *reinterpret_cast<int4*>(gs) = w;
                        gs[SW_OW] = sow;
                    }
                };
                if (lane < ns) put_state(succ);
                bool to_next = __any_sync(0xffffffffu, lane < ns && succ == i + 1);
                for (int k0 = 32; k0 < ns; k0 += 32) {
                    const int sr = k0 + lane < ns ? a.out_row[ra0.y + k0 + lane] : -1;
                    if (sr >= 0) put_state(sr);
                    to_next |= __any_sync(0xffffffffu, sr == i + 1);
                }
                if (to_next) {
                    nOl = sl >= 30 ? ol : mn(nOl, ol);
                    nOr = sl >= 30 ? orr : mx(nOr, orr);
                    nPl = mn(nPl, acj);
                    nPr = mx(nPr, acj + 1);
                    nOw = ow ? mx(nOw, ow) : ow;
                }
                if (lane == 0) {
                    sts32(slot(i) + 20, sl);
                    sts32(slot(i) + 24, acj);
                    a.state[8 * (int64_t)i + SW_SL] = sl;
                    a.state[8 * (int64_t)i + SW_MP] = acj;
                }
            }
            if (i + 1 < n) band_adaptive(rb0.z, rb0.w, m, a.w, nPl, nPr, nOl, nOr, nOw, Bs, Be);
        }
        __syncwarp();
        ra0 = rb0; ra1 = rb1; rb0 = rc0; rb1 = rc1;
        edx = edx_n; edx_n = edx_2;
        far = far_n; far_s = far_sn;
        succ = succ_n; succ_n = succ_2;
    }
    cells_out = cells;
    return ST_OK;
}

}  // namespace pb

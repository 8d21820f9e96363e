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
// bank conflicts).
//
// Measured on a B200 against the record fill it replaced (kernel time):
// 8,000 polishing windows 651 -> 339 ms, 1,024 windows of 2,000 bp at 15 %
// error with the adaptive band 1,118 -> 507 ms, one window of 64 reads 282 ->
// 131 ms. The fill's share of the polishing kernel fell from 62 % to 34 %.
#pragma once
#include "team.cuh"

namespace pb {

constexpr int WSTG = 16, WSTG_E = 64;  // rows and predecessor records staged at a time (static band)
constexpr int WSTG_BYTES = WSTG * 16 + WSTG_E * 16;
constexpr int WED = 32;                // an adaptive row's predecessor records in shared memory
// shared memory of the adaptive fill: records, then the state window
constexpr int warp_state_bytes(int rows) { return rows * SW_INTS * 4; }

struct WarpRing {
    unsigned at;  // shared memory address
    int rows;     // a power of two, or 0: no ring
    int blocks;   // per row
};

// One row. ed_at(e): {x, base in every byte, Bs, last block - Bs}, x the
// predecessor's ring offset (RING, -1: not in the ring, far(e) has its row-store
// block) or its row-store block. With ARGMAX, best / best_col become the row's
// first maximum.
template <bool WIDE, bool RING, bool ARGMAX, class EdAt, class Far>
__device__ __forceinline__ void warp_row(const CellK& k, int i, int Bs, int span, int tb, int d, const uint8_t* qs,
                                         const WarpRing& ring, char* store, int lane, EdAt ed_at, Far far, int32_t& best,
                                         int& best_col) {
    typedef Cells<WIDE> C;
    constexpr int32_t NEG = C::NEG;
    constexpr int32_t LOW = WIDE ? INT_MIN : -(1 << 30);
    constexpr int HB = 4 * C::BYTES, BB = 2 * HB;  // bytes per half block and block
    const int32_t g = k.o1 - k.e1;
    int32_t carry = add32(add32(NEG, k.e1), -k.o1);  // the gap term's floor: NEG_INF extended from column 0
    for (int c0 = 0; c0 <= span; c0 += 32) {
        const int b = c0 + lane, B = Bs + b;
        const bool act = b <= span;
        const int Bz = B == 0 ? INT_MAX : B;
        const uint2 qw = act ? *reinterpret_cast<const uint2*>(qs + (int64_t)B * BLK) : make_uint2(0x04040404u, 0x04040404u);
        int32_t P[8], V[8];
#pragma unroll
        for (int l = 0; l < 8; l++) P[l] = V[l] = NEG;
        if (i == 0 && B == 0) P[0] = 0;
        for (int e = 0; e < d; e++) {
            const int4 er = ed_at(e);
            const int pb = B - er.z;
            const bool in = act && (unsigned)pb <= (unsigned)er.w;
            const bool diag = in && Bz > er.z;  // the fill's block mask for the diagonal (src/align.cpp:1467)
            C lo, hi;
            lo.none();
            hi.none();
            int32_t left0 = NEG;  // lane 0: the cell before the chunk
            const bool l0 = lane == 0 && c0 > 0 && in && pb > 0;
            if (RING && er.x >= 0) {
                const unsigned src = ring.at + er.x + pb * HB;
                if (in) { lo.lds(src); hi.lds(src + ring.blocks * HB); }
                if (l0) left0 = C::lds_m(src + ring.blocks * HB - C::BYTES);
            } else {
                const char* src = store + ((int64_t)(RING ? far(e) : er.x) + pb) * BB;
                if (in) { lo.load(src); hi.load(src + HB); }
                if (l0) left0 = C::load_m(src - C::BYTES);
            }
            int32_t left = __shfl_up_sync(0xffffffffu, hi.m(3), 1);
            if (lane == 0) left = left0;  // (NEG_INF before the row's first block)
            const int32_t sm = diag || WIDE ? k.match : -(1 << 23), sx = diag || WIDE ? k.mismatch : -(1 << 23);
            const uint32_t x0 = qw.x ^ (uint32_t)er.y, x1 = qw.y ^ (uint32_t)er.y;
#pragma unroll
            for (int l = 0; l < 8; l++) {
                const int32_t src = l == 0 ? left : l <= 4 ? lo.m(l > 0 ? l - 1 : 0) : hi.m(l - 5);
                const int32_t cand = src + (((l < 4 ? x0 : x1) & (255u << (8 * (l & 3)))) == 0 ? sm : sx);
                if (!WIDE || diag) P[l] = mx(P[l], cand);
                V[l] = mx(V[l], l < 4 ? lo.v(l & 3, k) : hi.v(l & 3, k));
            }
        }
        int32_t H[8], key[8];
#pragma unroll
        for (int l = 0; l < 8; l++) {
            H[l] = mx(P[l], V[l]);
            key[l] = H[l] - l * k.e1;
        }
        const int32_t base = -(b * BLK) * k.e1;
        int32_t top = mx(mx(mx(key[0], key[1]), mx(key[2], key[3])), mx(mx(key[4], key[5]), mx(key[6], key[7])));
        const int32_t incl = scan_max(act ? top + base : LOW);
        int32_t ex = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) ex = LOW;
        if (ARGMAX) {
            // the first maximum of H0 is the row's first maximum (a gap never exceeds the cell it opens from)
            const int32_t lm = act ? mx(mx(mx(H[0], H[1]), mx(H[2], H[3])), mx(mx(H[4], H[5]), mx(H[6], H[7]))) : INT_MIN;
            const int32_t wm = __reduce_max_sync(0xffffffffu, lm);
            if (wm > best) {
                best = wm;
                int l = 7;
#pragma unroll
                for (int t = 6; t >= 0; t--) l = H[t] == wm ? t : l;
                best_col = __shfl_sync(0xffffffffu, B * BLK + l, __ffs(__ballot_sync(0xffffffffu, lm == wm)) - 1);
            }
        }
        int32_t run = mx(carry, ex) - base;
        carry = mx(carry, __shfl_sync(0xffffffffu, incl, 31));
        C lo, hi;
#pragma unroll
        for (int l = 0; l < 8; l++) {
            const int32_t M = i == 0 ? H[l] : mx(H[l], run + (g + l * k.e1));
            if (l < 4) lo.set(l & 3, M, V[l], k);
            else hi.set(l & 3, M, V[l], k);
            run = mx(run, key[l]);
        }
        if (act) {
            if (RING && span < ring.blocks) {
                const unsigned dst = ring.at + (i & (ring.rows - 1)) * (unsigned)(ring.blocks * BB) + b * HB;
                lo.sts(dst);
                hi.sts(dst + ring.blocks * HB);
            }
            char* dst = store + ((int64_t)tb + b) * BB;
            lo.store(dst);
            hi.store(dst + HB);
        }
    }
}

// Static band: rows and records staged WSTG rows at a time.
template <bool WIDE>
__device__ void warp_fill_static(const TeamJob& a, const WarpRing& ring, const uint8_t* qsm, unsigned char* stage, int lane) {
    const int n = a.n;
    const CellK k = a.k;
    char* const store = a.store;
    const unsigned stg = (unsigned)__cvta_generic_to_shared(stage);
    int32_t bm = 0;
    int bc = 0;
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
            const int4* far = a.ed;
            if (h.w & FR_UNSTAGED)
                warp_row<WIDE, true, false>(k, i, h.x, h.y, h.z, h.w & FR_D, qsm, ring, store, lane,
                                            [&](int e) { return fe[a.in_ptr[i] + e]; },
                                            [&](int e) { return far[a.in_ptr[i] + e].w; }, bm, bc);
            else
                warp_row<WIDE, true, false>(k, i, h.x, h.y, h.z, h.w & FR_D, qsm, ring, store, lane,
                                            [&](int e) { return lds128(ed + e * 16); },
                                            [&](int e) { return far[a.in_ptr[i] + e].w; }, bm, bc);
            __syncwarp();
        }
    }
}

// Adaptive band (-B) or full band (f = 0): bands known row by row. The band
// state's serial part is team_control's, on the same warp: inputs that do not
// need row i's maximum are fetched before the row is filled, the state of
// nearby rows lives in a shared-memory window of `wrows` rows (a power of two).
// Returns a status (uniform).
template <bool WIDE>
__device__ int warp_fill_dyn(const TeamJob& a, bool adaptive, unsigned char* wsm, int wrows, const uint8_t* qf, int lane,
                             int64_t& cells_out) {
    const int n = a.n, m = a.qlen + 1, E = a.in_ptr[n];
    const CellK k = a.k;
    char* const store = a.store;
    int4* sed = reinterpret_cast<int4*>(wsm);
    const unsigned seda = (unsigned)__cvta_generic_to_shared(wsm);
    int32_t* win = reinterpret_cast<int32_t*>(wsm + WED * 16);
    const int wmask = wrows - 1, AHEAD = wrows / 2 - 1;
    auto slot = [&](int r) { return win + (r & wmask) * SW_INTS; };
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
    if (lane < ra1.w) succ = a.out_row[ra0.y + lane];
    if (n > 1) {
        if (lane < rb1.z) edx_n = a.ed[rb0.x + lane].x;
        if (lane < rb1.w) succ_n = a.out_row[rb0.y + lane];
    }
    const WarpRing none{0, 0, 0};
    int32_t pend = 0;  // state entering the window, one int per lane (8)
    for (int i = 0; i < n; i++) {
        const int bn = Be - Bs - 1;
        const int d = i == 0 ? 0 : ra1.z, ns = ra1.w;
        if (bn < 0) return ST_DEGENERATE;
        if (d > MAX_MULTI_PRED) return ST_INDEGREE;
        if (tb + bn > a.store_cap || tb + bn > INT_MAX) return ST_OOM;
        // the state that entered the window after the previous row
        if (adaptive && i > 0 && i - 1 + AHEAD < n && lane < 8) slot(i - 1 + AHEAD)[lane] = pend;
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
        if (lane == 0) {
            a.rowi[i] = make_int4(Bs, Be, (int)tb, 0);
            int32_t* w = slot(i);
            w[SW_BS] = Bs; w[SW_BE] = Be; w[SW_TB] = (int)tb;
        }
        // row i's predecessor records; their slopes and maxima
        int psl = 0, pmp = INT_MIN / 2;
        for (int k0 = 0; k0 < d; k0 += 32) {
            const int kk = k0 + lane;
            if (kk < d) {
                int4 v;
                v.x = k0 == 0 ? edx : a.ed[ra0.x + kk].x;
                const int p = v.x >> 4;
                if (i - p < AHEAD) {
                    const int32_t* w = slot(p);
                    v.y = w[SW_BS]; v.z = w[SW_BE]; v.w = w[SW_TB];
                    if (k0 == 0) { psl = w[SW_SL]; pmp = w[SW_MP]; }
                } else {
                    const int4 q = a.rowi[p];
                    v.y = q.x; v.z = q.y; v.w = q.z;
                    if (adaptive && k0 == 0) { psl = a.state[8 * (int64_t)p + SW_SL]; pmp = a.state[8 * (int64_t)p + SW_MP]; }
                }
                if (kk < WED) sed[kk] = make_int4(v.w, (v.x & 7) * 0x01010101, v.y, v.z - 2 - v.y);
                a.ed[ra0.x + kk] = v;
            }
        }
        __syncwarp();
        int32_t* own = slot(i);
        const int32_t* nw = slot(i + 1);
        int sl = own[SW_SL], ow = own[SW_OW], ol = own[SW_OL], orr = own[SW_OR];
        int nPl = nw[SW_PL], nPr = nw[SW_PR], nOl = nw[SW_OL], nOr = nw[SW_OR], nOw = nw[SW_OW];
        const int4* ed = a.ed + ra0.x;
        auto ed_at = [&](int e) {
            if (e < WED) return lds128(seda + e * 16);
            const int4 v = ed[e];
            return make_int4(v.w, (v.x & 7) * 0x01010101, v.y, v.z - 2 - v.y);
        };
        auto far = [](int) { return 0; };
        int32_t best = INT_MIN;
        int acj = Bs * BLK;
        if (adaptive) warp_row<WIDE, false, true>(k, i, Bs, bn - 1, (int)tb, d, qf, none, store, lane, ed_at, far, best, acj);
        else warp_row<WIDE, false, false>(k, i, Bs, bn - 1, (int)tb, d, qf, none, store, lane, ed_at, far, best, acj);
        cells += (int64_t)bn * BLK;
        tb += bn;
        if (adaptive) {
            if (i >= 1) {  // src/align.cpp:1516-1568
                int sl_best = INT_MIN, max_slp = 0;
                bool is_match = false;
                if (ra1.y == (int)qf[acj + 1]) {  // cur.base == seq[max_acj]
                    max_slp = psl;
                    sl_best = pmp + 1 == acj ? psl + 1 : INT_MIN;
                    for (int kk = 32 + lane; kk < d; kk += 32) {
                        const int p = ed[kk].x >> 4;
                        const int32_t* w = i - p < AHEAD ? slot(p) : a.state + 8 * (int64_t)p;
                        max_slp = max(max_slp, w[SW_SL]);
                        if (w[SW_MP] + 1 == acj) sl_best = max(sl_best, w[SW_SL] + 1);
                    }
                    max_slp = __reduce_max_sync(0xffffffffu, max_slp);
                    sl_best = __reduce_max_sync(0xffffffffu, sl_best);
                    is_match = sl_best != INT_MIN;
                }
                if (is_match) sl = mx(sl, sl_best);
                if (!is_match && max_slp < 30) ow = mn(ow + max_slp + 1, 5 * a.w);
                if (sl >= 30) {
                    ol = orr = acj - ra1.x;
                    ow = 0;
                }
                bool to_next = false;
                for (int k0 = 0; k0 < ns; k0 += 32) {
                    const int kk = k0 + lane;
                    int sr = -1;
                    if (kk < ns) {
                        sr = k0 == 0 ? succ : a.out_row[ra0.y + kk];
                        int32_t* w = sr - i < AHEAD ? slot(sr) : a.state + 8 * (int64_t)sr;
                        w[SW_OL] = sl >= 30 ? ol : mn(w[SW_OL], ol);
                        w[SW_OR] = sl >= 30 ? orr : mx(w[SW_OR], orr);
                        w[SW_PL] = mn(w[SW_PL], acj);
                        w[SW_PR] = mx(w[SW_PR], acj + 1);
                        w[SW_OW] = ow ? mx(w[SW_OW], ow) : ow;
                    }
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
                    own[SW_SL] = sl; own[SW_MP] = acj;
                    a.state[8 * (int64_t)i + SW_SL] = sl;
                    a.state[8 * (int64_t)i + SW_MP] = acj;
                }
            }
            if (i + 1 < n) band_adaptive(rb0.z, rb0.w, m, a.w, nPl, nPr, nOl, nOr, nOw, Bs, Be);
        }
        __syncwarp();
        if (adaptive && i + AHEAD < n && lane < 8) pend = a.state[8 * (int64_t)(i + AHEAD) + lane];
        ra0 = rb0; ra1 = rb1; rb0 = rc0; rb1 = rc1;
        edx = edx_n; edx_n = edx_2;
        succ = succ_n; succ_n = succ_2;
    }
    cells_out = cells;
    return ST_OK;
}

}  // namespace pb

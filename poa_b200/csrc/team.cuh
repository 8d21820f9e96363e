// team.cuh - one banded POA alignment (one poa() call, src/align.cpp:1353-1737)
// by a team of warps: the DP fill, then the backtrack over the stored values.
//
// What bounds it: an alignment is a chain of dependent rows (one per graph
// rank), each only 30-200 blocks wide, so the time of one row step is the cost.
// Evaluating the backtrack's comparisons for every cell (the record fill of
// plain.cuh) made a row ~1,300 instructions per warp and ~4,300 cycles. Here
// the fill stores values instead and the backtrack compares only the cells it
// visits, which leaves ~15 integer operations per cell.
//
// Cells. A cell is stored as one 32-bit word, M << 8 | q, with
//   q = max(0, g - (M - D)),  g = max(e1 - o1, 1):
// the vertical term a successor takes is max(M + o1, D + e1) = M + o1 + q, and
// M == D iff q == g. A D so far below M that q is 0 can neither win a
// successor's maximum over M + o1 nor be a D the backtrack compares (it enters
// a D cell only through M == D, or by an extension that beat M + o1), so the
// word is an exact state, not an approximation. It needs |scores| < 2^20
// (cell_packable), with NEG in place of NEG_INF: unreachable cells lie in
// [NEG, NEG + 2^20], apart from every reachable value, and keep the
// reference's order and differences among themselves. Alignments beyond that
// range run the same code on {M, D} pairs (WIDE).
//
// Team. Columns are cut into strips of 128; strip s belongs to warp s % W, one
// thread per 4 cells (half a block). A thread meets the same columns in every
// row, so predecessor cells come back from the thread's own words in a
// shared-memory ring of the last TR rows (8 to 64, as many as fit; 16 bytes per
// thread, no bank conflicts) or, for rows further back, from the row store, and only the cell
// left of a strip crosses warps. Per row: predecessor pass, warp prefix
// maximum of the horizontal-gap keys, ONE barrier to exchange the warps'
// maxima, finalise, store. The left neighbour's last cell is derived from its
// published summary, so the next row does not wait for it to be stored.
// Rows wider than the team's 128 * W columns take several laps.
//
// Adaptive band: row i + 1's band depends on row i's first maximum. The first
// maximum of M is the first maximum of H0 = max(diagonal, vertical) (a gap
// never exceeds the cell it opens from), so it is published with the same
// barrier; two more warps, which own no columns, update the band state and
// prepare the next row's header while the others finalise the row.
//
// The row before is nearly always a predecessor; its cells stay in registers,
// so a row with no other predecessor reads no cells at all.
//
// Measured on a B200, DP kernels of one run, record fill -> this one: 10 reads
// of 16,569 bp, static band, 346 -> 125 ms (fill ~1,350 cycles per row of ~1,050
// cells, backtrack 325 cycles per move); 24 reads of 443 bp 31 -> 11 ms; 10
// reads of 5 kb at 10 % error, adaptive band, 308 -> 92 ms; 840 seeded
// sub-windows 94 -> 27 ms. What is left is latency: ~215 mostly dependent
// instructions per warp and row.
#pragma once
#include <type_traits>

#include "plain.cuh"

namespace pb {

struct CellK {
    int32_t match, mismatch, o1, e1;
    int32_t gq;      // max(e1 - o1, 1)
    uint32_t qmask;  // 255, or 0 when e1 == o1 (no extension beats a new gap)
};

PB_HD CellK cell_consts(const Scoring& s) {
    CellK k;
    k.match = s.match; k.mismatch = s.mismatch; k.o1 = s.o1; k.e1 = s.e1;
    const int32_t g = s.e1 - s.o1;
    k.gq = g > 1 ? g : 1;
    k.qmask = g > 0 ? 255u : 0u;
    return k;
}

// The packed cell holds every alignment of up to n rows and m columns.
PB_HD bool cell_packable(const Scoring& s, int64_t n, int64_t m) {
    int64_t big = 1;
    const int64_t v[4] = {s.match, s.mismatch, s.o1, s.e1};
    for (int k = 0; k < 4; k++) {
        const int64_t a = v[k] < 0 ? -v[k] : v[k];
        if (a > big) big = a;
    }
    const bool bytes = s.match >= -128 && s.match <= 127 && s.mismatch >= -128 && s.mismatch <= 127;  // score_table
    return bytes && big < (1 << 20) && (n + m + 2) * big < (1 << 20) && (int64_t)s.e1 - s.o1 <= 255;
}

// Scores of a predecessor's base against query codes 0..3, one byte each; code 4
// (N) matches base 4 only, whose table is the mismatch in every byte.
PB_HD uint32_t score_table(const CellK& k, int base) {
    const uint32_t x = ((uint32_t)k.mismatch & 255u) * 0x01010101u;
    return base < 4 ? x ^ ((((uint32_t)k.match ^ (uint32_t)k.mismatch) & 255u) << (8 * base)) : x;
}

constexpr int32_t PACK_NEG = -(1 << 22);

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ int4 lds128(unsigned a) {
    int4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ int32_t lds32(unsigned a) {
    int32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts32(unsigned a, int32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts128(unsigned a, int4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ int lds_u16(unsigned a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int lds_u8(unsigned a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return (int)v;
}
__device__ __forceinline__ void sts_u16(unsigned a, int v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void sts_u8(unsigned a, int v) {
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

template <bool WIDE> struct Cells;

template <> struct Cells<false> {
    static constexpr int32_t NEG = PACK_NEG;
    static constexpr int BYTES = 4;
    int32_t c[4];
    __device__ __forceinline__ void none() { c[0] = c[1] = c[2] = c[3] = NEG * 256; }
    __device__ __forceinline__ void load(const void* p) {
        const int4 v = *reinterpret_cast<const int4*>(p);
        c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
    }
    __device__ __forceinline__ void store(void* p) const {
        *reinterpret_cast<int4*>(p) = make_int4(c[0], c[1], c[2], c[3]);
    }
    __device__ __forceinline__ void lds(unsigned a) {
        const int4 v = lds128(a);
        c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
    }
    __device__ __forceinline__ void sts(unsigned a) const { sts128(a, make_int4(c[0], c[1], c[2], c[3])); }
    static __device__ __forceinline__ int32_t lds_m(unsigned a) { return lds32(a) >> 8; }
    static __device__ __forceinline__ int32_t load_m(const void* p) { return *reinterpret_cast<const int32_t*>(p) >> 8; }
    __device__ __forceinline__ int32_t m(int l) const { return c[l] >> 8; }
    // vertical terms are kept less o1: max(M + o1, D + e1) - o1
    __device__ __forceinline__ int32_t v(int l, const CellK& k) const {
        return (c[l] >> 8) + (int32_t)((uint32_t)c[l] & k.qmask);
    }
    __device__ __forceinline__ void set(int l, int32_t M, int32_t V, const CellK& k) {
        c[l] = (int32_t)((uint32_t)M << 8) + mx(V - M + (k.gq + k.o1), 0);
    }
    // one cell of the row store, for the backtrack
    struct One {
        int32_t w;
        static __device__ __forceinline__ One lds(unsigned a) { return One{lds32(a)}; }
        __device__ __forceinline__ int32_t m() const { return w >> 8; }
        __device__ __forceinline__ bool eq_md(const CellK& k) const { return (w & 255) == k.gq; }
        __device__ __forceinline__ bool d_opens(int32_t d, const CellK& k) const { return m() + k.o1 == d; }
        __device__ __forceinline__ bool d_extends(int32_t d, const CellK& k) const {
            const int32_t q = (int32_t)((uint32_t)w & k.qmask);
            return q > 0 && m() + k.o1 + q == d;
        }
    };
};

template <> struct Cells<true> {
    static constexpr int32_t NEG = NEG_INF;
    static constexpr int BYTES = 8;
    int32_t M_[4], D_[4];
    __device__ __forceinline__ void none() {
#pragma unroll
        for (int l = 0; l < 4; l++) M_[l] = D_[l] = NEG;
    }
    __device__ __forceinline__ void load(const void* p) {
        const int4 a = reinterpret_cast<const int4*>(p)[0], b = reinterpret_cast<const int4*>(p)[1];
        M_[0] = a.x; D_[0] = a.y; M_[1] = a.z; D_[1] = a.w;
        M_[2] = b.x; D_[2] = b.y; M_[3] = b.z; D_[3] = b.w;
    }
    __device__ __forceinline__ void store(void* p) const {
        reinterpret_cast<int4*>(p)[0] = make_int4(M_[0], D_[0], M_[1], D_[1]);
        reinterpret_cast<int4*>(p)[1] = make_int4(M_[2], D_[2], M_[3], D_[3]);
    }
    __device__ __forceinline__ void lds(unsigned a) {
        const int4 u = lds128(a), v = lds128(a + 16);
        M_[0] = u.x; D_[0] = u.y; M_[1] = u.z; D_[1] = u.w;
        M_[2] = v.x; D_[2] = v.y; M_[3] = v.z; D_[3] = v.w;
    }
    __device__ __forceinline__ void sts(unsigned a) const {
        sts128(a, make_int4(M_[0], D_[0], M_[1], D_[1]));
        sts128(a + 16, make_int4(M_[2], D_[2], M_[3], D_[3]));
    }
    static __device__ __forceinline__ int32_t lds_m(unsigned a) { return lds32(a); }
    static __device__ __forceinline__ int32_t load_m(const void* p) { return *reinterpret_cast<const int32_t*>(p); }
    __device__ __forceinline__ int32_t m(int l) const { return M_[l]; }
    __device__ __forceinline__ int32_t v(int l, const CellK& k) const { return mx(M_[l], D_[l] + (k.e1 - k.o1)); }
    __device__ __forceinline__ void set(int l, int32_t M, int32_t V, const CellK& k) { M_[l] = M; D_[l] = V + k.o1; }
    struct One {
        int32_t M, D;
        static __device__ __forceinline__ One lds(unsigned a) { return One{lds32(a), lds32(a + 4)}; }
        __device__ __forceinline__ int32_t m() const { return M; }
        __device__ __forceinline__ bool eq_md(const CellK&) const { return M == D; }
        __device__ __forceinline__ bool d_opens(int32_t d, const CellK& k) const { return add32(M, k.o1) == d; }
        __device__ __forceinline__ bool d_extends(int32_t d, const CellK& k) const { return add32(D, k.e1) == d; }
    };
};

// One alignment's rows and buffers (device pointers).
struct TeamJob {
    int32_t n, qlen, f, w;   // rows, query length, band parameters (w = b + m / f)
    CellK k;
    const int32_t* in_ptr;   // [n + 1] predecessors of each row
    // [edges] in the backtrack's priority order (in_weight descending, in-list
    // position ascending): x = predecessor row << 4 | (in_weight >= ind / 10) << 3
    // | its base as the DP sees it; y, z, w = its band and row-store block,
    // filled in here
    int4* ed;
    int4* fe;                // [edges] the same for the fill, the row before left out: {ring offset, or ~row-store block; base in every byte; Bs; last block - Bs}
    const int32_t *hq, *tq;  // [n] static band
    const int4* ra;          // [2 n] adaptive band: {first in-edge, first out-edge, hq, tq}, {hq_loc, base, d, successors}
    const int32_t* out_row;  // adaptive band: successor rows in out-list order
    const uint8_t* qs;       // shifted query (dp_job.h)
    int4* rowi;              // [n] {Bs, Be, row-store block, -}
    int4* fr;                // [n] static band, for the fill: {Bs, last block - Bs, row-store block, d | flags | first record in the stage}
    int32_t* state;          // [8 n] adaptive band state of rows outside the shared-memory window
    char* store;             // cells, 8 per block
    int64_t store_cap;       // blocks
    int32_t* moves;
    int32_t moves_cap;
    int32_t* out;            // [0] status, [1] score, [2] moves, [3] cells
};

constexpr int TC = 4;           // cells per thread
constexpr int STRIP = 32 * TC;  // columns per warp
constexpr int SBLK = STRIP / BLK;
constexpr int STG = 32;         // rows staged at a time (static band)
constexpr int STG_E = 128;      // their predecessor records
constexpr int HDR_E = 32;       // predecessor records in an adaptive row's header
constexpr int SWIN = 256;       // rows of the adaptive state window (a power of two), half of them ahead
constexpr int SW_INTS = 12;     // {Pl, Pr, Ol, Or, Ow, Sl, Mp, -, Bs, Be, tb, -}
enum { SW_PL = 0, SW_PR, SW_OL, SW_OR, SW_OW, SW_SL, SW_MP, SW_BS = 8, SW_BE, SW_TB };
// flags in a row header's last word: listed predecessors in the low 10 bits;
// FR_PREV: the row before is a predecessor too, its base above FR_PBASE
enum { FR_D = 1023, FR_GENERAL = 1 << 10, FR_UNSTAGED = 1 << 11, FR_PREV = 1 << 12, FR_PBASE = 13, FR_EOFF = 16 };

struct TeamStage {
    int4 row[STG];
    int4 ed[STG_E];
};
struct TeamHdr {
    int4 h;        // {Bs, last block - Bs, row-store block, FR_GENERAL | status << FR_EOFF}
    int4 g;        // {first in-edge, predecessors, flags and count of the fill's list, -}
    int4 ed[HDR_E];  // the fill's list, as TeamJob::fe
};

// Backtrack tile (team_backtrack): up to BT_ROWS rows around the walk, as many
// as `bytes` of shared memory hold, BLKS blocks of each, their rows, their
// predecessor records and where their heaviest predecessors lead.
constexpr int BT_ROWS = 64;

template <bool WIDE, int BLKS>
struct BtTile {
    static constexpr int ROWB = BLKS * BLK * Cells<WIDE>::BYTES;
    static constexpr int PER_ROW = ROWB + 16 + 3 * 16 + 4 + 5;
    int rows, E;              // rows and predecessor records
    int row, ed, ptr, jump;   // byte offsets: int4 {Bs, Be, store block, first block of the tile row}; int4; int; uint8 [5][rows]
    __host__ __device__ explicit BtTile(int bytes) {
        const int r = (bytes - 16) / PER_ROW;
        rows = r < BT_ROWS ? r : BT_ROWS;
        E = 3 * rows;
        row = rows * ROWB;
        ed = row + rows * 16;
        ptr = ed + E * 16;
        jump = ptr + (rows + 4) * 4;
    }
    static constexpr int full() { return BT_ROWS * PER_ROW + 16; }
};

// RING_MAX: shared memory for the ring of rows (one CTA per SM by default).
constexpr int RING_ALONE = 196608;
template <int W, bool ADAPT, bool WIDE, int RING_MAX = RING_ALONE>
struct TeamSmem {
    static constexpr int CELLB = TC * Cells<WIDE>::BYTES;          // bytes per thread and row
    static constexpr int ROWB = 32 * W * CELLB;
    // rows of the ring (a power of two): noisy graphs have predecessors tens of rows back, and
    // one read from the row store costs as much as a row
    static constexpr int TR = ROWB * 64 <= RING_MAX ? 64 : ROWB * 32 <= RING_MAX ? 32 : ROWB * 16 <= RING_MAX ? 16 : 8;
    static constexpr int RING = TR * ROWB;
    static constexpr int PUB = RING;                               // int4 [2][W]
    static constexpr int BEST = PUB + 2 * W * 16;                  // int4 [2][W]
    static constexpr int REST = BEST + 2 * W * 16;
    static constexpr int FILL =
        REST + (ADAPT ? 2 * (int)sizeof(TeamHdr) + SWIN * SW_INTS * 4 : 2 * (int)sizeof(TeamStage));
    static constexpr int BYTES = FILL > BtTile<WIDE, 8>::full() ? FILL : BtTile<WIDE, 8>::full();
    static constexpr int THREADS = 32 * (W + (ADAPT ? 2 : 0));
};

// Named barriers: 1 the whole team, 2 the compute warps' maxima (they arrive,
// the state warp waits), 3 the compute warps.
template <int ID, int NT>
__device__ __forceinline__ void bar_sync() { asm volatile("barrier.sync %0, %1;" ::"n"(ID), "n"(NT) : "memory"); }
template <int ID, int NT>
__device__ __forceinline__ void bar_arrive() { asm volatile("barrier.arrive %0, %1;" ::"n"(ID), "n"(NT) : "memory"); }

// Inclusive prefix maximum over the warp in three rounds of independent
// shuffles (a lane without a source gets its own value back, which a maximum
// does not mind).
__device__ __forceinline__ int32_t scan_max(int32_t v) {
    const int32_t a = __shfl_up_sync(0xffffffffu, v, 1), b = __shfl_up_sync(0xffffffffu, v, 2),
                  c = __shfl_up_sync(0xffffffffu, v, 3);
    v = mx(mx(v, a), mx(b, c));
    const int32_t d = __shfl_up_sync(0xffffffffu, v, 4), e = __shfl_up_sync(0xffffffffu, v, 8),
                  f = __shfl_up_sync(0xffffffffu, v, 12);
    v = mx(mx(v, d), mx(e, f));
    return mx(v, __shfl_up_sync(0xffffffffu, v, 16));
}

// A predecessor's band as the fill's records hold it, {Bs, last block - Bs}: an
// empty band as one block that no row reaches.
__device__ __forceinline__ int2 rec_band(int Bs, int Be) {
    return Be - 2 - Bs >= 0 ? make_int2(Bs, Be - 2 - Bs) : make_int2(1 << 29, 0);
}

__device__ __forceinline__ int strips_of(int Bs, int Be) { return ((Be - 2) >> 4) - (Bs >> 4) + 1; }

// Static band: every row's band and place in the row store, its header for
// the fill, and each predecessor record's copy of its row's. Returns a status
// (uniform).
template <class S, int W, int NT>
__device__ int team_rows_static(const TeamJob& a, int64_t* s_part, unsigned long long* s_fail, int64_t& cells) {
    const int tid = threadIdx.x, n = a.n, m = a.qlen + 1;
    if (tid == 0) *s_fail = ~0ull;
    __syncthreads();
    int64_t run = 0;
    for (int r0 = 0; r0 < n; r0 += NT) {
        const int i = r0 + tid;
        int Bs = 0, Be = 1, d = 0;
        if (i < n) {
            band_static(a.f, a.hq[i], a.tq[i], m, a.w, Bs, Be);
            if (i == 0) Bs = 0;
            d = i == 0 ? 0 : a.in_ptr[i + 1] - a.in_ptr[i];
        }
        const int bn = Be - Bs - 1;
        int64_t v = i < n && bn > 0 ? bn : 0, total;
        // CTA-wide exclusive prefix sum
        const int lane = tid & 31, wid = tid >> 5;
        int64_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_part[wid] = x;
        __syncthreads();
        int64_t before = 0;
        total = 0;
        for (int k = 0; k < NT / 32; k++) {
            const int64_t p = s_part[k];
            if (k < wid) before += p;
            total += p;
        }
        __syncthreads();
        const int64_t off = run + before + x - v;
        run += total;
        if (i < n) {
            int st = ST_OK;
            if (bn < 0) st = ST_DEGENERATE;
            else if (d > MAX_MULTI_PRED) st = ST_INDEGREE;
            else if (off + bn > a.store_cap || off + bn > INT_MAX) st = ST_OOM;
            if (st != ST_OK) atomicMin(s_fail, ((unsigned long long)i << 8) | (unsigned long long)st);
            a.rowi[i] = make_int4(Bs, Be, (int)off, 0);
        }
    }
    __syncthreads();
    cells = run * BLK;
    if (*s_fail != ~0ull) return (int)(*s_fail & 255ull);
    for (int i = tid; i < n; i += NT) {
        const int4 ri = a.rowi[i];
        const int e0 = a.in_ptr[i], d = i == 0 ? 0 : a.in_ptr[i + 1] - e0;
        const int eoff = e0 - a.in_ptr[i & ~(STG - 1)];
        int fl = d;
        if (i == 0 || ri.y - ri.x - 1 <= 0 || strips_of(ri.x, ri.y) > W) fl |= FR_GENERAL;
        if (eoff + d > STG_E) fl |= FR_UNSTAGED;
        else fl |= eoff << FR_EOFF;
        int x = e0;
        for (int e = e0; e < e0 + d; e++) {
            int4 v = a.ed[e];
            const int p = v.x >> 4;
            const int4 pr = a.rowi[p];
            v.y = pr.x; v.z = pr.y; v.w = pr.z;
            a.ed[e] = v;
            const bool lap1 = pr.y - pr.x - 1 > 0 && strips_of(pr.x, pr.y) <= W;
            if (lap1 && p == i - 1 && !(fl & FR_GENERAL)) fl += FR_PREV - 1 + ((v.x & 7) << FR_PBASE);
            else {
                const int2 band = rec_band(pr.x, pr.y);
                a.fe[x++] = make_int4(lap1 && i - p < S::TR ? (p & (S::TR - 1)) * S::ROWB : ~pr.z, (v.x & 7) * 0x01010101, band.x,
                                      band.y);
            }
        }
        a.fr[i] = make_int4(ri.x, ri.y - 2 - ri.x, ri.z, fl);
    }
    __syncthreads();
    return ST_OK;
}

template <int W>
__device__ __forceinline__ void team_stage(const TeamJob& a, TeamStage& st, int i0) {
    // rows [i0, i0 + STG) and their predecessor records, by the whole CTA
    const int tid = threadIdx.x, n = a.n;
    const int cnt = min(STG, n - i0);
    if (cnt <= 0) return;
    const int e0 = a.in_ptr[i0], ne = min(a.in_ptr[i0 + cnt] - e0, STG_E);
    for (int x = tid; x < cnt; x += 32 * W) cp_async16(&st.row[x], a.fr + i0 + x);
    for (int x = tid; x < ne; x += 32 * W) cp_async16(&st.ed[x], a.fe + e0 + x);
    cp_async_commit_all();
}

// The fill of one row by a column-owning thread; see the file comment.
template <int W, bool ADAPT, bool WIDE, int RING_MAX = RING_ALONE>
struct TeamRow {
    typedef Cells<WIDE> C;
    typedef TeamSmem<W, ADAPT, WIDE, RING_MAX> S;
    static constexpr int32_t NEG = C::NEG;
    static constexpr int32_t LOW = WIDE ? INT_MIN : -(1 << 30);
    const TeamJob& a;
    const CellK k;
    char* const store;
    const unsigned sb, own, leftw;  // shared memory: base, this thread's cells, the word left of them (within a ring row)
    const int lane, wid;
    const int32_t K;                // the gap term's floor: NEG_INF extended from column 0
    int s_cur = INT_MIN / 2;        // this warp's strip
    int col0 = 0, B = 0, Bz = 0;    // its first column, block (and that block, or a large value for block 0: no diagonal mask there)
    uint32_t qw = 0;                // query codes of the thread's columns
    int qn = 4;                     // code of the column after them (adaptive band)
    // the row before, when it fits the team's columns: band, this thread's M and vertical
    // terms (VNEG outside the band), M left of the thread's columns
    int pBs = 0, pspan = -1;
    const int32_t VNEG;             // NEG_INF as a vertical term (less o1)
    int32_t pm[4], pe[4], pleft = C::NEG;
    unsigned xp = 0;                // byte offset of the published summaries' half in use

    __device__ TeamRow(char* sm, const TeamJob& job)
        : a(job), k(job.k), store(job.store), sb((unsigned)__cvta_generic_to_shared(sm)),
          own(threadIdx.x * S::CELLB), leftw((threadIdx.x == 0 ? 32 * W : threadIdx.x) * S::CELLB - C::BYTES),
          lane(threadIdx.x & 31), wid(threadIdx.x >> 5), K(add32(add32(C::NEG, job.k.e1), -job.k.o1)),
          VNEG(C::NEG - job.k.o1) {
#pragma unroll
        for (int l = 0; l < 4; l++) { pm[l] = NEG; pe[l] = VNEG; }
    }

    __device__ __forceinline__ void take_strip(int s) {
        s_cur = s;
        col0 = s * STRIP + lane * TC;
        B = col0 >> 3;
        Bz = B == 0 ? INT_MAX : B;
        const bool in = col0 + 8 <= (int)qs_bytes(a.qlen);
        qw = in ? *reinterpret_cast<const uint32_t*>(a.qs + col0) : 0x04040404u;
        if (ADAPT) qn = in ? a.qs[col0 + 4] : 4;
        // the row before had other columns here, if any
#pragma unroll
        for (int l = 0; l < 4; l++) { pm[l] = NEG; pe[l] = VNEG; }
    }

    // diagonal terms of one predecessor: m its M, left the M before them
    __device__ __forceinline__ void diagonal(const int32_t* m, int32_t left, bool diag, uint32_t x, int32_t* P) const {
        // packed cells: a term pushed far below NEG drops out of the maximum
        const int32_t sm = diag || WIDE ? k.match : -(1 << 23), sx = diag || WIDE ? k.mismatch : -(1 << 23);
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const int32_t cand = (l == 0 ? left : m[l > 0 ? l - 1 : 0]) + ((x & (255u << (8 * l))) == 0 ? sm : sx);
            if (!WIDE || diag) P[l] = mx(P[l], cand);
        }
    }
    __device__ __forceinline__ void fold(const C& pc, int32_t left, bool diag, uint32_t x, int32_t* P, int32_t* V) const {
        const int32_t m[4] = {pc.m(0), pc.m(1), pc.m(2), pc.m(3)};
        diagonal(m, left, diag, x, P);
#pragma unroll
        for (int l = 0; l < 4; l++) V[l] = mx(V[l], pc.v(l, k));
    }

    // prefix maximum within the warp and its summary; base: -(column in the row's band) * e1
    __device__ __forceinline__ void publish(bool act, const int32_t* H, int32_t base, int32_t* key, int32_t& ex) const {
        key[0] = H[0];
        key[1] = H[1] - k.e1;
        key[2] = H[2] - 2 * k.e1;
        key[3] = H[3] - 3 * k.e1;
        const int32_t k02 = mx(mx(key[0], key[1]), key[2]);
        const int32_t incl = scan_max(act ? mx(k02, key[3]) + base : LOW);
        ex = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) ex = LOW;
        if (lane == 31)
            sts128(sb + S::PUB + xp + wid * 16, make_int4(incl, act ? mx(ex, k02 + base) : ex, H[3], s_cur));
    }
    __device__ __forceinline__ void publish_none() const {
        if (lane == 31) sts128(sb + S::PUB + xp + wid * 16, make_int4(LOW, LOW, NEG, INT_MAX));
    }
    // the row's first maximum so far in this warp: value, column, and the query code after that column
    __device__ __forceinline__ void maximum(bool act, const int32_t* H, int4& best) const {
        const int32_t lm = act ? mx(mx(H[0], H[1]), mx(H[2], H[3])) : INT_MIN;
        const int32_t wm = __reduce_max_sync(0xffffffffu, lm);
        if (wm > best.x) {
            const int first = __ffs(__ballot_sync(0xffffffffu, lm == wm)) - 1;
            const int l = H[0] == wm ? 0 : H[1] == wm ? 1 : H[2] == wm ? 2 : 3;
            const int code = l == 3 ? qn : (int)((qw >> (8 * (l + 1))) & 255u);
            const int v = __shfl_sync(0xffffffffu, (col0 + l) * 8 + code, first);
            best = make_int4(wm, v >> 3, v & 7, 0);
        }
    }
    __device__ __forceinline__ void put_maximum(const int4& best) const {
        if (lane == 0) sts128(sb + S::BEST + xp + wid * 16, best);
        __syncwarp();
        bar_arrive<2, 32 * (W + 1)>();
    }
    // M of the thread's cells (into H) from the prefix maximum `run` left of them
    __device__ __forceinline__ void gaps(int32_t* H, const int32_t* key, int32_t run) const {
        const int32_t g = k.o1 - k.e1;
        H[0] = mx(H[0], run + g);
        run = mx(run, key[0]);
        H[1] = mx(H[1], run + (g + k.e1));
        run = mx(run, key[1]);
        H[2] = mx(H[2], run + (g + 2 * k.e1));
        run = mx(run, key[2]);
        H[3] = mx(H[3], run + (g + 3 * k.e1));
    }
    // stores the thread's cells and keeps the row as the row before of the next;
    // edge: M of the cell left of the strip
    __device__ __forceinline__ void keep(int i, const int4& h, bool act, const int32_t* M, const int32_t* V, int rel, int32_t edge) {
        if (act) {
            C o;
#pragma unroll
            for (int l = 0; l < 4; l++) o.set(l, M[l], V[l], k);
            o.sts(sb + (i & (S::TR - 1)) * S::ROWB + own);
            o.store(store + ((int64_t)h.z * BLK + rel) * C::BYTES);
        }
#pragma unroll
        for (int l = 0; l < 4; l++) {
            pm[l] = M[l];
            pe[l] = act ? mx(M[l], add32(V[l], k.e1)) : VNEG;
        }
        pleft = __shfl_up_sync(0xffffffffu, M[3], 1);
        if (lane == 0) pleft = edge;
    }
    __device__ __forceinline__ void sync_row() const {
        if (ADAPT) bar_sync<3, 32 * W>();
        else bar_sync<1, S::THREADS>();
    }

    // A row that fits the team's columns (i > 0). ed_at(e): the e-th listed record.
    template <class EdAt, class After>
    __device__ __forceinline__ void row(int i, int4 h, EdAt ed_at, After after_barrier) {
        const int Bs = h.x, span = h.y, d = h.w & FR_D;
        const int S0 = Bs >> 4, S1 = (Bs + span) >> 4;
        if ((unsigned)(s_cur - S0) >= (unsigned)W) {
            int r = (wid - S0) % W;
            take_strip(S0 + (r < 0 ? r + W : r));
        }
        const bool on = s_cur <= S1;
        const int rel = col0 - Bs * BLK;
        const bool act = on && (unsigned)(B - Bs) <= (unsigned)span;
        const bool first = B == Bs && !(lane & 1);  // column 0 of the row's first block reads NEG_INF
        int32_t P[4], V[4], H[4], key[4], ex = LOW, base = 0;
        if (on) {
#pragma unroll
            for (int l = 0; l < 4; l++) { P[l] = NEG; V[l] = VNEG; }
            if (h.w & FR_PREV) {
                // diag: the fill's block mask for the diagonal (src/align.cpp:1467)
                const bool diag = (unsigned)(B - pBs) <= (unsigned)pspan && Bz > pBs;
                diagonal(pm, first ? NEG : pleft, diag, qw ^ (((uint32_t)h.w >> FR_PBASE & 7u) * 0x01010101u), P);
#pragma unroll
                for (int l = 0; l < 4; l++) V[l] = mx(VNEG, pe[l]);
            }
            if (d > 0) __syncwarp();  // the ring's words of the lanes to the left
            for (int e = 0; e < d; e++) {
                const int4 er = ed_at(e);
                const bool in = (unsigned)(B - er.z) <= (unsigned)er.w;
                const bool diag = in && Bz > er.z;
                C pc;
                int32_t left;
                if (er.x >= 0) {
                    pc.lds(sb + er.x + own);
                    left = C::lds_m(sb + er.x + leftw);
                    if (!in) pc.none();
                } else {
                    const char* src = store + ((int64_t)~er.x * BLK + (col0 - er.z * BLK)) * C::BYTES;
                    pc.none();
                    left = NEG;
                    if (in && act) {
                        pc.load(src);
                        if (B > er.z || (lane & 1)) left = C::load_m(src - C::BYTES);
                    }
                }
                if (first) left = NEG;
                fold(pc, left, diag, qw ^ (uint32_t)er.y, P, V);
            }
#pragma unroll
            for (int l = 0; l < 4; l++) H[l] = mx(P[l], add32(V[l], k.o1));
            if (ADAPT) {
                int4 best = make_int4(INT_MIN, 0, 0, 0);
                maximum(act, H, best);
                put_maximum(best);
            }
            base = -rel * k.e1;
            publish(act, H, base, key, ex);
        } else {
            if (ADAPT) put_maximum(make_int4(INT_MIN, 0, 0, 0));
            publish_none();
        }
        sync_row();
        after_barrier();
        pBs = Bs;
        pspan = span;
        if (on) {
            const int4 pv = lane < W ? lds128(sb + S::PUB + xp + lane * 16) : make_int4(LOW, LOW, NEG, INT_MAX);
            const int4 L = lds128(sb + S::PUB + xp + (wid == 0 ? W - 1 : wid - 1) * 16);
            const int32_t Pl = mx(K, __reduce_max_sync(0xffffffffu, pv.w < s_cur - 1 ? pv.x : LOW));
            const int32_t Pr = s_cur > S0 ? mx(Pl, L.x) : Pl;
            // M of the cell left of the strip (lane 0's), from its warp's summary
            const int32_t edge = mx(L.z, add32(k.o1 + (rel - 2) * k.e1, mx(Pl, L.y)));
            gaps(H, key, mx(Pr, ex) - base);
            keep(i, h, act, H, V, rel, edge);
        } else {
#pragma unroll
            for (int l = 0; l < 4; l++) pe[l] = VNEG;
        }
        xp ^= W * 16;
    }

    // Row 0, and rows wider than the team's columns: laps of W strips, every
    // predecessor cell from the row store, and a barrier at the end of the row.
    __device__ __forceinline__ void general(int i, int4 h, const int4* ed) {
        const int Bs = h.x, bn = h.y + 1, d = h.w & FR_D;
        const int S0 = Bs >> 4, S1 = bn > 0 ? (Bs + h.y) >> 4 : S0 - 1;
        const int laps = S1 - S0 + 1 > W ? (S1 - S0 + W) / W : 1;
        int r = (wid - S0) % W;
        if (r < 0) r += W;
        int32_t carry = K;
        int4 best = make_int4(INT_MIN, Bs * BLK, 4, 0);
        for (int c = 0; c < laps; c++) {
            const int s = S0 + c * W + r;
            const bool on = s <= S1;
            int32_t P[4], V[4], H[4], key[4], ex = LOW, base = 0;
            bool act = false;
            int rel = 0;
            if (on) {
                if (s != s_cur) take_strip(s);
                act = B >= Bs && B <= Bs + h.y;
                rel = col0 - Bs * BLK;
#pragma unroll
                for (int l = 0; l < 4; l++) { P[l] = NEG; V[l] = VNEG; }
                if (i == 0 && col0 == 0) P[0] = 0;
                for (int e = 0; e < d; e++) {
                    const int4 fe = ed[e];
                    const bool in = act && B >= fe.y && B <= fe.z - 2;
                    const bool diag = in && (B > fe.y || B == 0);
                    C pc;
                    pc.none();
                    int32_t left = NEG;
                    if (in) {
                        const char* src = store + ((int64_t)fe.w * BLK + (col0 - fe.y * BLK)) * C::BYTES;
                        pc.load(src);
                        if ((B > fe.y || (lane & 1)) && !(B == Bs && !(lane & 1))) left = C::load_m(src - C::BYTES);
                    }
                    fold(pc, left, diag, qw ^ (uint32_t)((fe.x & 7) * 0x01010101), P, V);
                }
#pragma unroll
                for (int l = 0; l < 4; l++) H[l] = mx(P[l], add32(V[l], k.o1));
                base = -rel * k.e1;
                publish(act, H, base, key, ex);
                if (ADAPT) maximum(act, H, best);
            } else {
                publish_none();
            }
            if (ADAPT && c == laps - 1) put_maximum(best);
            sync_row();
            const int4 pv = lane < W ? lds128(sb + S::PUB + xp + lane * 16) : make_int4(LOW, LOW, NEG, INT_MAX);
            const int32_t P0 = mx(carry, __reduce_max_sync(0xffffffffu, pv.w < s ? pv.x : LOW));
            const int32_t Pl = mx(K, __reduce_max_sync(0xffffffffu, pv.w < s - 1 ? pv.x : LOW));
            carry = mx(carry, __reduce_max_sync(0xffffffffu, pv.x));
            if (on) {
                if (i > 0) gaps(H, key, mx(P0, ex) - base);
                if (S1 - S0 < W) {
                    const int4 L = lds128(sb + S::PUB + xp + (wid == 0 ? W - 1 : wid - 1) * 16);
                    keep(i, h, act, H, V, rel, i == 0 ? L.z : mx(L.z, add32(k.o1 + (rel - 2) * k.e1, mx(Pl, L.y))));
                } else if (act) {
                    C o;
#pragma unroll
                    for (int l = 0; l < 4; l++) o.set(l, H[l], V[l], k);
                    o.store(store + ((int64_t)h.z * BLK + rel) * C::BYTES);
                }
            } else {
#pragma unroll
                for (int l = 0; l < 4; l++) pe[l] = VNEG;
            }
            xp ^= W * 16;
        }
        pBs = Bs;
        pspan = h.y;
        if (!ADAPT) sync_row();
    }
};

template <int W, bool WIDE>
__device__ void team_fill_static(const TeamJob& a, char* smem) {
    typedef TeamSmem<W, false, WIDE> S;
    TeamRow<W, false, WIDE> t(smem, a);
    TeamStage* stage = reinterpret_cast<TeamStage*>(smem + S::REST);
    const unsigned stg = (unsigned)__cvta_generic_to_shared(stage);
    team_stage<W>(a, stage[0], 0);
    cp_async_wait_all();
    bar_sync<1, S::THREADS>();
    const int n = a.n;
    int4 h = lds128(stg);
    bool unpublished = false;  // the row before stored its cells after its barrier
    for (int i = 0; i < n; i++) {
        const int x = i & (STG - 1);
        const unsigned cur = stg + ((i / STG) & 1) * (unsigned)sizeof(TeamStage);
        if (x == 0) team_stage<W>(a, stage[((i / STG) & 1) ^ 1], i + STG);
        if (x == STG - 1) cp_async_wait_all();  // the next stage, published by this row's barrier
        const unsigned nxt = x == STG - 1 ? stg + (((i / STG) & 1) ^ 1) * (unsigned)sizeof(TeamStage) : cur + (x + 1) * 16;
        if (h.w & FR_GENERAL) {
            // reads every predecessor from the row store, the row before's among them
            if (unpublished) t.sync_row();
            t.general(i, h, a.ed + a.in_ptr[i]);
            unpublished = false;
            h = lds128(nxt);
        } else {
            unpublished = true;
            const int4 hc = h;
            const unsigned ed = cur + STG * 16 + (hc.w >> FR_EOFF) * 16;
            t.row(i, hc, [&](int e) { return hc.w & FR_UNSTAGED ? a.fe[a.in_ptr[i] + e] : lds128(ed + e * 16); },
                  [&]() { h = lds128(nxt); });
        }
    }
    __syncthreads();
}

// The adaptive band's serial part (src/align.cpp:1433-1444, 1516-1568) on two
// warps of its own. The state warp turns a row's maximum into the next row's
// band; the records warp prepares the next row's predecessor records. Rows' state
// and places live in a shared-memory window of SWIN rows around the current one
// (successors up to SWIN / 2 - 2 rows ahead, predecessors up to SWIN / 2
// behind), in global memory beyond it. Between the row's maxima and the next
// header there is only what depends on them; everything else runs while the
// other warps fill the row. (As one warp the two took 2,400 cycles a row.)
// Lists are one pass for up to 32 entries that reads the window whatever the row,
// the state 16 bytes at a time: as loops around the near / far branch the noisy 5 kb
// graph's kernel took 101 ms, now 92.
constexpr int AHEAD = SWIN / 2 - 1;

template <int W, bool WIDE, int RING_MAX = RING_ALONE>
__device__ void team_state(const TeamJob& a, char* smem, int64_t& cells_out) {
    typedef TeamSmem<W, true, WIDE, RING_MAX> S;
    TeamHdr* hdr = reinterpret_cast<TeamHdr*>(smem + S::REST);
    const unsigned win = (unsigned)__cvta_generic_to_shared(smem + S::REST + 2 * sizeof(TeamHdr));
    const unsigned bests = (unsigned)__cvta_generic_to_shared(smem + S::BEST);
    const int lane = threadIdx.x & 31;
    const int n = a.n, m = a.qlen + 1, E = a.in_ptr[n], bw = a.w;
    const int4* ra = a.ra;
    const int4* ed = a.ed;
    const int32_t* out_row = a.out_row;
    int32_t* state = a.state;
    const int64_t store_cap = a.store_cap;
    // row r's state: {Pl, Pr, Ol, Or}, {Ow, Sl, Mp, -}, {Bs, Be, tb, -}
    auto slot = [&](int r) { return win + (r & (SWIN - 1)) * (SW_INTS * 4); };
    int4 ra0 = ra[0], ra1 = ra[1];                // row i
    int4 rb0 = make_int4(0, 0, 0, 0), rb1 = rb0;  // row i + 1
    if (n > 1) { rb0 = ra[2]; rb1 = ra[3]; }
    int Bs, Be;
    band_adaptive(ra0.z, ra0.w, m, bw, m, 0, 0, 0, 0, Bs, Be);
    Bs = 0;
    int64_t tb = 0, cells = 0;
    // the header's band, place, and (last word) GENERAL or a failed status
    auto put_header = [&](int i, int d) {
        const int bn = Be - Bs - 1;
        int st = ST_OK;
        if (bn < 0) st = ST_DEGENERATE;
        else if (d > MAX_MULTI_PRED) st = ST_INDEGREE;
        else if (tb + bn > store_cap || tb + bn > INT_MAX) st = ST_OOM;
        const bool gen = i == 0 || bn <= 0 || strips_of(Bs, Be) > W;
        if (lane == 0) hdr[i & 1].h = make_int4(Bs, Be - 2 - Bs, (int)tb, (gen ? FR_GENERAL : 0) | (st << FR_EOFF));
        return st;
    };
    int st = put_header(0, 0);
    int edx = 0, edx_n = 0;      // row i's and row i + 1's predecessor records (x), one per lane
    int succ = -1, succ_n = -1;  // their successors, one per lane
    if (lane < ra1.w) succ = out_row[ra0.y + lane];
    if (n > 1) {
        if (lane < rb1.z) edx_n = ed[rb0.x + lane].x;
        if (lane < rb1.w) succ_n = out_row[rb0.y + lane];
    }
    int2 far_s = make_int2(0, 0);  // row i's predecessors beyond the window: slope and maximum, one per lane
    __syncwarp();
    bar_sync<1, S::THREADS>();  // header 0
    int xp = 0;
    for (int i = 0; i < n; i++) {
        if (st != ST_OK) {
            if (lane == 0) a.out[0] = st;
            cells_out = cells;
            return;
        }
        const int bn = Be - Bs - 1;
        const int d = i == 0 ? 0 : ra1.z, ns = ra1.w;
        if (lane == 0) {
            a.rowi[i] = make_int4(Bs, Be, (int)tb, 0);
            sts128(slot(i) + 32, make_int4(Bs, Be, (int)tb, 0));
        }
        int32_t pend = 0;  // state entering the window, one int per lane (8)
        if (i > 0 && i - 1 + AHEAD < n && lane < 8) pend = state[8 * (int64_t)(i - 1 + AHEAD) + lane];
        // loads two rows ahead
        int4 rc0 = rb0, rc1 = rb1;
        int edx_2 = 0, succ_2 = -1;
        if (i + 2 < n) {
            rc0 = ra[2 * (i + 2)];
            rc1 = ra[2 * (i + 2) + 1];
            // (the in-window in-edges and out-edges are the same edges: E of each)
            const int e2 = rb0.x + rb1.z, o2 = rb0.y + rb1.w;
            if (e2 + lane < E) edx_2 = ed[e2 + lane].x;
            if (o2 + lane < E) succ_2 = out_row[o2 + lane];
        }
        int2 far_n = make_int2(0, 0);
        if (lane < rb1.z && i + 1 - (edx_n >> 4) >= AHEAD) {
            const int32_t* w = state + 8 * (int64_t)(edx_n >> 4);
            far_n = make_int2(w[SW_SL], w[SW_MP]);
        }
        // row i's predecessors' slopes and maxima (their rows are done), its own
        // state and the next row's
        int psl = 0, pmp = INT_MIN / 2;
        if (lane < d) {
            const int p = edx >> 4;
            const int4 w = lds128(slot(p) + 16);
            psl = i - p < AHEAD ? w.y : far_s.x;
            pmp = i - p < AHEAD ? w.z : far_s.y;
        }
        int max_psl = psl, pmp0 = pmp;
        if (d > 1) {
            max_psl = __reduce_max_sync(0xffffffffu, psl);
        } else {
            max_psl = __shfl_sync(0xffffffffu, psl, 0);
            pmp0 = __shfl_sync(0xffffffffu, pmp, 0);
        }
        const int4 own0 = lds128(slot(i)), own1 = lds128(slot(i) + 16), nw = lds128(slot(i + 1));
        int sl = own1.y, ow = own1.x, ol = own0.z, orr = own0.w;
        int nPl = nw.x, nPr = nw.y, nOl = nw.z, nOr = nw.w, nOw = lds32(slot(i + 1) + 16);
        bool to_next = __any_sync(0xffffffffu, lane < ns && succ == i + 1);
        for (int k0 = 32; k0 < ns; k0 += 32)
            to_next |= __any_sync(0xffffffffu, k0 + lane < ns && out_row[ra0.y + k0 + lane] == i + 1);
        // the row's maxima: published in the last lap's half of the summaries
        const int nst = bn > 0 ? strips_of(Bs, Be) : 0;
        const int laps = nst > W ? (nst + W - 1) / W : 1;
        xp = (xp + laps - 1) & 1;
        // the state that enters the window
        if (i > 0 && i - 1 + AHEAD < n && lane < 8) sts32(slot(i - 1 + AHEAD) + 4 * lane, pend);
        __syncwarp();
        bar_sync<2, 32 * (W + 1)>();
        int acj = 0;
        if (i >= 1) {
            const int4 bq = lane < W ? lds128(bests + (xp * W + lane) * 16) : make_int4(INT_MIN, 0, 0, 0);
            const int32_t best = __reduce_max_sync(0xffffffffu, bq.x);
            const int key = __reduce_min_sync(0xffffffffu, bq.x == best ? bq.y * 8 + bq.z : INT_MAX);
            acj = bn > 0 ? key >> 3 : Bs * BLK;
            const int code = bn > 0 ? key & 7 : (int)a.qs[acj + 1];
            int sl_best = INT_MIN, max_slp = 0;
            if (ra1.y == code) {  // cur.base == seq[max_acj]
                max_slp = max_psl;
                if (d <= 1) {
                    if (pmp0 + 1 == acj) sl_best = max_psl + 1;
                } else if (d <= 32) {
                    sl_best = __reduce_max_sync(0xffffffffu, pmp + 1 == acj ? psl + 1 : INT_MIN);
                } else {
                    for (int kk = lane; kk < d; kk += 32) {
                        const int p = ed[ra0.x + kk].x >> 4;
                        const int4 w = i - p < AHEAD ? lds128(slot(p) + 16)
                                                     : *reinterpret_cast<const int4*>(state + 8 * (int64_t)p + 4);
                        max_slp = max(max_slp, w.y);
                        if (w.z + 1 == acj) sl_best = max(sl_best, w.y + 1);
                    }
                    max_slp = __reduce_max_sync(0xffffffffu, max_slp);
                    sl_best = __reduce_max_sync(0xffffffffu, sl_best);
                }
            }
            const bool is_match = sl_best != INT_MIN;
            if (is_match) sl = mx(sl, sl_best);
            else if (max_slp < 30) ow = mn(ow + max_slp + 1, 5 * bw);
            if (sl >= 30) {
                ol = orr = acj - ra1.x;
                ow = 0;
            }
            if (to_next) {
                nOl = sl >= 30 ? ol : mn(nOl, ol);
                nOr = sl >= 30 ? orr : mx(nOr, orr);
                nPl = mn(nPl, acj);
                nPr = mx(nPr, acj + 1);
                nOw = ow ? mx(nOw, ow) : ow;
            }
        }
        cells += (int64_t)bn * BLK;
        tb += bn;
        if (i + 1 < n) {
            band_adaptive(rb0.z, rb0.w, m, bw, nPl, nPr, nOl, nOr, nOw, Bs, Be);
            st = put_header(i + 1, rb1.z);
        }
        __syncwarp();
        bar_sync<1, S::THREADS>();  // header i + 1; row i's cells
        if (i >= 1) {
            if (lane == 0) {
                sts32(slot(i) + 20, sl);
                sts32(slot(i) + 24, acj);
                int32_t* gs = state + 8 * (int64_t)i;
                gs[SW_SL] = sl; gs[SW_MP] = acj;
            }
            auto put_state = [&](int sr) {
                const bool near = sr - i < AHEAD;
                int32_t* gs = state + 8 * (int64_t)sr;
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
            for (int kk = 32 + lane; kk < ns; kk += 32) put_state(out_row[ra0.y + kk]);
        }
        __syncwarp();
        xp ^= 1;
        far_s = far_n;
        ra0 = rb0; ra1 = rb1; rb0 = rc0; rb1 = rc1;
        edx = edx_n; edx_n = edx_2;
        succ = succ_n; succ_n = succ_2;
    }
    cells_out = cells;
}

// Row i + 1's records while row i is filled: every predecessor's band and place
// (TeamJob::ed), and the fill's list, without row i when that fits the team's
// columns (TeamHdr).
template <int W, bool WIDE, int RING_MAX = RING_ALONE>
__device__ void team_records(const TeamJob& a, char* smem) {
    typedef TeamSmem<W, true, WIDE, RING_MAX> S;
    TeamHdr* hdr = reinterpret_cast<TeamHdr*>(smem + S::REST);
    const unsigned win = (unsigned)__cvta_generic_to_shared(smem + S::REST + 2 * sizeof(TeamHdr));
    const unsigned hb = (unsigned)__cvta_generic_to_shared(hdr);
    const int lane = threadIdx.x & 31;
    const int n = a.n, E = a.in_ptr[n];
    int4* ed = a.ed;
    int4* fe = a.fe;
    const int32_t* in_ptr = a.in_ptr;
    // row i + 1: first in-edge, end, and the records (x) one per lane; row i + 2's are fetched a row ahead
    int e0 = n > 1 ? in_ptr[1] : 0, e1 = n > 1 ? in_ptr[2] : 0, e2 = n > 2 ? in_ptr[3] : e1;
    int x = e0 + lane < E ? ed[e0 + lane].x : 0;
    if (lane == 0) hdr[0].g = make_int4(0, 0, 0, 0);
    __syncwarp();
    bar_sync<1, S::THREADS>();  // header 0
    for (int i = 0; i < n; i++) {
        const int4 h = lds128(hb + (i & 1) * (unsigned)sizeof(TeamHdr));
        if (h.w >> FR_EOFF) return;
        const int x2 = e1 + lane < E ? ed[e1 + lane].x : 0;
        const int e3 = i + 4 <= n ? in_ptr[i + 4] : e2;
        if (i + 1 < n) {
            TeamHdr& o = hdr[(i + 1) & 1];
            const int Bs = h.x, Be = h.x + h.y + 2, dn = e1 - e0;
            const bool lap1 = h.y >= 0 && strips_of(Bs, Be) <= W;
            int prev = 0;
            auto put = [&](int k0, int vx) {
                const int kk = k0 + lane, p = vx >> 4;
                const bool has = kk < dn, own = has && p == i;
                int4 q = make_int4(0, 0, 0, 0);  // its band and place
                if (has) {
                    q = lds128(win + (p & (SWIN - 1)) * (SW_INTS * 4) + 32);
                    if (i - p >= AHEAD) q = a.rowi[p];
                    if (own) q = make_int4(Bs, Be, h.z, 0);
                    ed[e0 + kk] = make_int4(vx, q.x, q.y, q.z);
                }
                const unsigned pmask = __ballot_sync(0xffffffffu, lap1 && own);
                if (has && !((pmask >> lane) & 1u)) {
                    const int at = kk - (prev != 0 || (pmask & ((1u << lane) - 1u)) != 0);
                    const bool near = i + 1 - p < S::TR && q.y - q.x - 1 > 0 && strips_of(q.x, q.y) <= W;
                    const int2 band = rec_band(q.x, q.y);
                    const int4 f = make_int4(near ? (p & (S::TR - 1)) * S::ROWB : ~q.z, (vx & 7) * 0x01010101, band.x, band.y);
                    if (at < HDR_E) o.ed[at] = f;
                    else fe[e0 + at] = f;
                }
                if (pmask) prev = FR_PREV | ((__shfl_sync(0xffffffffu, vx, __ffs(pmask) - 1) & 7) << FR_PBASE);
            };
            if (dn > 0) put(0, x);
            for (int k0 = 32; k0 < dn; k0 += 32) put(k0, k0 + lane < dn ? ed[e0 + k0 + lane].x : 0);
            // {first in-edge, predecessors, the fill's flags and count, -}
            if (lane == 0) o.g = make_int4(e0, dn, (dn - (prev != 0)) | prev, 0);
        }
        __syncwarp();
        bar_sync<1, S::THREADS>();  // header i + 1
        e0 = e1; e1 = e2; e2 = e3;
        x = x2;
    }
}

template <int W, bool WIDE, int RING_MAX = RING_ALONE>
__device__ int team_fill_adaptive(const TeamJob& a, char* smem, int64_t& cells) {
    typedef TeamSmem<W, true, WIDE, RING_MAX> S;
    const int tid = threadIdx.x, n = a.n, m = a.qlen + 1;
    int32_t* win = reinterpret_cast<int32_t*>(smem + S::REST + 2 * sizeof(TeamHdr));
    TeamHdr* hdr = reinterpret_cast<TeamHdr*>(smem + S::REST);
    for (int64_t x = tid; x < 8 * (int64_t)n; x += S::THREADS) a.state[x] = (x & 7) == SW_PL ? m : 0;
    for (int x = tid; x < SWIN * SW_INTS; x += S::THREADS) win[x] = x % SW_INTS == SW_PL ? m : 0;
    if (tid == 0) a.out[0] = ST_OK;
    bar_sync<1, S::THREADS>();
    if (tid >= 32 * (W + 1)) {
        team_records<W, WIDE, RING_MAX>(a, smem);
    } else if (tid >= 32 * W) {
        team_state<W, WIDE, RING_MAX>(a, smem, cells);
    } else {
        TeamRow<W, true, WIDE, RING_MAX> t(smem, a);
        const unsigned hb = (unsigned)__cvta_generic_to_shared(hdr);
        bar_sync<1, S::THREADS>();  // header 0
        for (int i = 0; i < n; i++) {
            const unsigned hc = hb + (i & 1) * (unsigned)sizeof(TeamHdr);
            int4 h = lds128(hc);
            const int4 g = lds128(hc + 16);
            if (h.w >> FR_EOFF) break;
            if (h.w & FR_GENERAL) {
                h.w |= g.y;
                t.general(i, h, a.ed + g.x);
            } else {
                h.w = g.z;
                t.row(i, h, [&](int e) { return e < HDR_E ? lds128(hc + 32 + e * 16) : a.fe[g.x + e]; }, [] {});
            }
            bar_sync<1, S::THREADS>();  // row i's cells, header i + 1
        }
    }
    __syncthreads();
    return a.out[0];
}

// Backtrack by one warp over the stored values, src/align.cpp:1572-1736: the
// same steps, tests and tie rules as backtrack_records (dp_rowops.h), each test
// evaluated on the cells the walk reaches, one lane per predecessor (they are
// in priority order, so "the first that passes" is a ballot).
//
// A step is a chain of dependent reads and ~100 dependent instructions (1,250
// cycles measured), so
//  * what it reads comes from a tile in shared memory: BT_ROWS rows up to the
//    walk's, for each its predecessor records and BT_BLK blocks around the
//    column the walk would reach if it kept its distance from the band's left
//    end. Cells outside the tile are read from the row store; a walk that
//    leaves its row's blocks, or the tile's first row, loads the next tile;
//  * runs of matches along the heaviest in-edges are taken in one step: lane t
//    stands t such predecessors back (pointer jumping over the tile's rows) and
//    t columns to the left, and tests whether its cell's first choice, a match
//    with its heaviest predecessor, holds. The leading lanes' moves are the
//    walk's. The cell that ends the run takes the full step.
//
// M == I is decided only when it is asked for, by looking for the cell the
// gap opened from: I[j] is the maximum over k < j of M[k] + o1 + (j - 1 - k) * e1
// and never exceeds M[j]. Once in a gap the walk carries the gap's value.
//
// Loading a tile was the walk's largest part (10,400 cycles for 64 rows, most of
// it one row's chain of address arithmetic after another): two rows a lane, the
// rows' cells 8 passes in flight and the jump tables from registers through
// 32-bit shared-memory addresses take 6,300. The search for a gap's origin goes
// 128 columns and then 384 at a time: 2,860 -> 1,300 cycles on 12 kb rows.
// ROOMY: builds with the registers for that. Those that share the SM with three
// or four more CTAs of 4 warps keep 2 passes and 128 columns: full unrolling
// spills there (8,000 polishing windows: 233 ms against 209; before, 214).
template <bool WIDE, int BT_BLK, bool ROOMY = true>
static __device__ __noinline__ int32_t team_backtrack(const TeamJob& a, char* smem, int bytes, int lane, int32_t& nmoves) {
    typedef typename Cells<WIDE>::One One;
    const BtTile<WIDE, BT_BLK> T(bytes);
    constexpr int ROWB = BtTile<WIDE, BT_BLK>::ROWB, BACK = BT_BLK - (BT_BLK >= 8 ? 3 : 2);  // blocks kept left of the walk's
    constexpr int32_t NEG = Cells<WIDE>::NEG;
    constexpr int CB = Cells<WIDE>::BYTES, RL = ROWB / 16;  // 16-byte pieces of a tile row
    const CellK k = a.k;
    const One* store = reinterpret_cast<const One*>(a.store);
    const int4* rowi = a.rowi;
    const int4* edg = a.ed;
    const uint8_t* qs = a.qs;
    int32_t* moves = a.moves;
    const int cap = a.moves_cap;
    const unsigned sb = (unsigned)__cvta_generic_to_shared(smem);
    int i = a.n - 1, acj = a.qlen + 1, op = ALL_OP;
    int32_t carry = 0;  // the value of the gap the walk is in (op == D_OP or I_OP)
    int32_t nm = 0;
    int lo = INT_MAX, e_lo = 0, ne = 0;
    int32_t st = ST_OK;
    while (i > 0 || acj > 0) {
        int4 R = make_int4(0, 0, 0, 0);
        if (i >= lo) R = lds128(sb + T.row + (i - lo) * 16);
        if (i < lo || (unsigned)((acj >> 3) - R.w) >= BT_BLK) {
            // the tile that ends with row i
            lo = max(0, i - T.rows + 1);
            const int cnt = i - lo + 1;
            const int dB = (acj >> 3) - rowi[i].x;
            __syncwarp();
            // rows and list ends: two rows a lane
            int4 v[2];
            int ends[3];
#pragma unroll
            for (int q = 0; q < 2; q++) v[q] = lane + 32 * q < cnt ? rowi[lo + lane + 32 * q] : make_int4(0, 0, 0, 0);
#pragma unroll
            for (int q = 0; q < 3; q++) ends[q] = lane + 32 * q <= cnt ? a.in_ptr[lo + lane + 32 * q] : 0;
            e_lo = __shfl_sync(0xffffffffu, ends[0], 0);
            {
                const int x0 = __shfl_sync(0xffffffffu, ends[0], cnt & 31), x1 = __shfl_sync(0xffffffffu, ends[1], cnt & 31),
                          x2 = __shfl_sync(0xffffffffu, ends[2], cnt & 31);
                ne = min((cnt < 32 ? x0 : cnt < 64 ? x1 : x2) - e_lo, T.E);
            }
            for (int e = lane; e < ne; e += 32) cp_async16(smem + T.ed + e * 16, edg + e_lo + e);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                v[q].w = v[q].x + max(0, dB - BACK);
                if (lane + 32 * q < cnt) sts128(sb + T.row + (lane + 32 * q) * 16, v[q]);
            }
#pragma unroll
            for (int q = 0; q < 3; q++)
                if (lane + 32 * q <= cnt) *reinterpret_cast<int32_t*>(smem + T.ptr + (lane + 32 * q) * 4) = ends[q];
            __syncwarp();
            constexpr int RPI = 32 / RL, TU = ROOMY ? 8 : 2;  // rows a pass takes, passes in flight
            for (int r0 = lane / RL; r0 < cnt; r0 += RPI * TU) {
                int4 w[TU];
#pragma unroll
                for (int q = 0; q < TU; q++) w[q] = r0 + RPI * q < cnt ? lds128(sb + T.row + (r0 + RPI * q) * 16) : make_int4(0, 0, 0, 0);
#pragma unroll
                for (int q = 0; q < TU; q++) {
                    const int r = r0 + RPI * q, pc = lane % RL;
                    if (r < cnt && w[q].w + pc * 16 / (BLK * CB) <= w[q].y - 2)
                        cp_async16(smem + r * ROWB + pc * 16, a.store + ((int64_t)w[q].z + (w[q].w - w[q].x)) * (BLK * CB) + pc * 16);
                }
            }
            cp_async_commit_all();
            cp_async_wait_all();
            __syncwarp();
            // where the heaviest predecessors lead, 1, 2, 4, 8 and 16 steps back
            int to[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int r = lane + 32 * q;
                to[q] = 255;
                if (r < cnt && lo + r > 0) {
                    const int e = lds32(sb + T.ptr + r * 4) - e_lo, e1 = lds32(sb + T.ptr + r * 4 + 4) - e_lo;
                    if (e < e1 && e < ne) {
                        const int p = lds32(sb + T.ed + e * 16) >> 4;
                        if (p >= lo) to[q] = p - lo;
                    }
                }
                if (r < T.rows) sts_u8(sb + T.jump + r, to[q]);
            }
#pragma unroll
            for (int x = 1; x < 5; x++) {
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 2; q++)
                    to[q] = to[q] == 255 ? 255 : lds_u8(sb + T.jump + (x - 1) * T.rows + to[q]);
#pragma unroll
                for (int q = 0; q < 2; q++)
                    if (lane + 32 * q < T.rows) sts_u8(sb + T.jump + x * T.rows + lane + 32 * q, to[q]);
            }
            __syncwarp();
            R = lds128(sb + T.row + (i - lo) * 16);
        }
        if (op & M_OP) {
            // a run of matches with the heaviest predecessors
            int r = i - lo;
#pragma unroll
            for (int q = 0; q < 5; q++)
                if (((lane >> q) & 1) && r != 255) r = lds_u8(sb + T.jump + q * T.rows + r);
            const int c = acj - lane;
            bool ok = false;
            int32_t mv = 0;
            const int to = r == 255 ? 255 : lds_u8(sb + T.jump + r);
            if (to != 255 && c > 0) {
                const int4 A = lds128(sb + T.row + r * 16), P = lds128(sb + T.row + to * 16);
                const int4 er = lds128(sb + T.ed + (lds32(sb + T.ptr + r * 4) - e_lo) * 16);
                const int qc = qs[c], bl = (c - 1) >> 3;
                // both cells in their rows' bands and in the tile
                if ((c >> 3) <= A.y - 2 && (unsigned)((c >> 3) - A.w) < BT_BLK && bl <= P.y - 2 && (unsigned)(bl - P.w) < BT_BLK &&
                    (er.x & 15) == (qc | 8)) {
                    const int32_t x = One::lds(sb + r * ROWB + (c - A.w * BLK) * CB).m();
                    const int32_t y = One::lds(sb + to * ROWB + (c - 1 - P.w * BLK) * CB).m();
                    ok = x == add32(y, k.match);
                    mv = mv_pack(MV_MATCH, lo + to, qc);
                }
            }
            const unsigned bad = ~__ballot_sync(0xffffffffu, ok);
            const int run = min(bad ? __ffs(bad) - 1 : 32, cap - nm);
            if (run > 0) {
                if (lane < run) moves[nm + lane] = mv;
                nm += run;
                acj -= run;
                op = ALL_OP;
                i = __shfl_sync(0xffffffffu, to, run - 1) + lo;
                continue;
            }
        }
        const int Bs = R.x, Be = R.y;
        if (acj > (Be - 1) * BLK || acj < Bs * BLK) { st = ST_BAND_ESCAPE; break; }
        const int j = acj - Bs * BLK;
        if (j >= (Be - Bs - 1) * BLK) { st = ST_BT_FAIL; break; }
        if (nm + 1 > cap) { st = ST_OOM; break; }
        const int e0 = lds32(sb + T.ptr + (i - lo) * 4) - e_lo;
        const int d = i == 0 ? 0 : lds32(sb + T.ptr + (i - lo) * 4 + 4) - e_lo - e0;
        const One cell = One::lds(sb + (i - lo) * ROWB + (acj - R.w * BLK) * CB);
        const int qc = acj > 0 ? qs[acj] : 4;
        const int32_t M = cell.m();
        const bool eq_md = cell.eq_md(k);
        const int32_t dv = op == D_OP ? carry : M;
        int p1 = -1, p4 = -1, po = -1, pe = -1;  // rows of the choices; p1 -2: the heaviest match fails its weight test
        bool m4_match = false;
        for (int k0 = 0; k0 < d; k0 += 32) {
            bool em = false, bm = false, eo = false, ex = false;
            int4 er = make_int4(0, 0, 0, 0);
            if (k0 + lane < d) {
                const int e = e0 + k0 + lane;
                if (e < ne) er = lds128(sb + T.ed + e * 16);
                else er = edg[e_lo + e];
                const int p = er.x >> 4;
                const int bl = (acj - 1) >> 3, bc = acj >> 3;
                const bool inl = acj > 0 && bl >= er.y && bl <= er.z - 2;
                const bool inc = bc >= er.y && bc <= er.z - 2;
                int w0 = INT_MIN / 2;
                if (p >= lo) w0 = lds32(sb + T.row + (p - lo) * 16 + 12);
                One vl, vc;
                if (inl) {
                    if ((unsigned)(bl - w0) < BT_BLK) vl = One::lds(sb + (p - lo) * ROWB + (acj - 1 - w0 * BLK) * CB);
                    else vl = store[(int64_t)er.w * BLK + (acj - 1 - er.y * BLK)];
                }
                if (inc) {
                    if ((unsigned)(bc - w0) < BT_BLK) vc = One::lds(sb + (p - lo) * ROWB + (acj - w0 * BLK) * CB);
                    else vc = store[(int64_t)er.w * BLK + (acj - er.y * BLK)];
                    eo = vc.d_opens(dv, k);
                    ex = vc.d_extends(dv, k);
                }
                if (inl) {
                    bm = (er.x & 7) == qc;
                    em = M == add32(vl.m(), bm ? k.match : k.mismatch);
                }
            }
            const unsigned b1 = __ballot_sync(0xffffffffu, em && bm);
            if (b1 && p1 == -1) {
                const int x = __shfl_sync(0xffffffffu, er.x, __ffs(b1) - 1);
                p1 = (x & 8) ? x >> 4 : -2;
                if (p1 >= 0 && (op & M_OP) && acj > 0 && k0 == 0) break;  // the walk's first choice
            }
            const unsigned b4 = __ballot_sync(0xffffffffu, em), bo = __ballot_sync(0xffffffffu, eo),
                           be = __ballot_sync(0xffffffffu, ex);
            if (b4 && p4 < 0) {
                const int f = __ffs(b4) - 1;
                p4 = __shfl_sync(0xffffffffu, er.x, f) >> 4;
                m4_match = (b1 >> f) & 1;
            }
            if (bo && po < 0) po = __shfl_sync(0xffffffffu, er.x, __ffs(bo) - 1) >> 4;
            if (be && pe < 0) pe = __shfl_sync(0xffffffffu, er.x, __ffs(be) - 1) >> 4;
        }
        if ((op & M_OP) && acj > 0 && p1 >= 0) {
            if (lane == 0) moves[nm] = mv_pack(MV_MATCH, p1, qc);
            nm++;
            op = ALL_OP; i = p1; acj--;
            continue;
        }
        if ((op & D_OP) && (op == D_OP || eq_md) && (po >= 0 || pe >= 0)) {
            if (po >= 0) { i = po; op = M_OP | I_OP; }
            else { i = pe; op = D_OP; carry = add32(dv, -k.e1); }
            continue;
        }
        if ((op & I_OP) && acj > 0 && j >= 1) {
            const One* row = store + (int64_t)R.z * BLK;
            bool in_gap = op == I_OP;
            int32_t v = carry;
            if (!in_gap) {  // M == I ?
                v = M;
                if (i == 0) {
                    in_gap = M == NEG;
                } else {
                    // 128 columns, then more at a time (a round trip to the row store each)
                    constexpr int FAR = ROOMY ? 12 : 4;
                    auto look = [&](int x0, auto n) {
                        One c[decltype(n)::value];
                        bool hit = false;
#pragma unroll
                        for (int u = 0; u < decltype(n)::value; u++)
                            if (x0 - 32 * u - lane >= 0) c[u] = row[x0 - 32 * u - lane];
#pragma unroll
                        for (int u = 0; u < decltype(n)::value; u++) {
                            const int x = x0 - 32 * u - lane;
                            if (x >= 0) hit |= add32(c[u].m(), k.o1 + (j - 1 - x) * k.e1) == v;
                        }
                        return __any_sync(0xffffffffu, hit) != 0;
                    };
                    in_gap = look(j - 1, std::integral_constant<int, 4>());
                    for (int x0 = j - 129; x0 >= 0 && !in_gap; x0 -= 32 * FAR) in_gap = look(x0, std::integral_constant<int, FAR>());
                    in_gap = in_gap || add32(NEG, j * k.e1) == v;
                }
            }
            if (in_gap) {
                const bool iopen = add32(row[j - 1].m(), k.o1) == v;
                const bool iext = i > 0 || k.e1 == 0;  // I is one or the other; row 0 holds NEG throughout
                if (iopen || iext) {
                    if (lane == 0) moves[nm] = mv_pack(MV_INSERT, 0, qc);
                    nm++;
                    if (iopen) op = M_OP | D_OP;
                    else { op = I_OP; carry = add32(v, -k.e1); }
                    acj--;
                    continue;
                }
            }
        }
        if ((op & M_OP) && acj > 0 && p4 >= 0) {
            if (lane == 0) moves[nm] = mv_pack(m4_match ? MV_MATCH : MV_MISMATCH, p4, qc);
            nm++;
            op = ALL_OP; i = p4; acj--;
            continue;
        }
        st = ST_BT_FAIL;
        break;
    }
    nmoves = nm;
    return st;
}

// Score, status and moves of a filled alignment (warp 0).
template <bool WIDE, int BLKS>
static __device__ void team_finish(const TeamJob& a, char* smem, int bytes, int64_t cells, int lane) {
    const int m = a.qlen + 1;
    int32_t nm = 0;
    const int32_t st = team_backtrack<WIDE, BLKS>(a, smem, bytes, lane, nm);
    if (lane == 0) {
        const int4 last = a.rowi[a.n - 1];
        const int jm = m - last.x * BLK;
        // column m lies in the last row's band (tlen[end] - tlen[end] = 0); the
        // guard only keeps a malformed window from reading outside its row
        const bool inb = jm >= 0 && jm / BLK < last.y - last.x - 1;
        int32_t score = NEG_INF;
        if (inb) {
            score = reinterpret_cast<const typename Cells<WIDE>::One*>(a.store)[(int64_t)last.z * BLK + jm].m();
            if (!WIDE && score < -(1 << 21)) score += NEG_INF - PACK_NEG;  // an unreachable end cell
        }
        a.out[1] = score;
        a.out[2] = nm;
        a.out[3] = (int32_t)(cells > INT_MAX ? INT_MAX : cells);
        a.out[0] = st;
    }
}

// One CTA per alignment.
template <int W, bool ADAPT, bool WIDE>
__global__ void __launch_bounds__(TeamSmem<W, ADAPT, WIDE>::THREADS, 1) k_align(const TeamJob* __restrict__ jobs) {
    typedef TeamSmem<W, ADAPT, WIDE> S;
    extern __shared__ __align__(16) char tsm[];
    __shared__ TeamJob sa;
    __shared__ int64_t s_part[W + 1];
    __shared__ unsigned long long s_fail;
    __shared__ int64_t s_cells;
    if (threadIdx.x == 0) sa = jobs[blockIdx.x];
    __syncthreads();
    const TeamJob& a = sa;
    int64_t cells = 0;
    if (a.n <= 0) {
        if (threadIdx.x == 0) a.out[0] = ST_BAD_ARG;
        return;
    }
    int st;
    if constexpr (ADAPT) {
        st = team_fill_adaptive<W, WIDE>(a, tsm, cells);
        if (threadIdx.x == 32 * W) s_cells = cells;  // the state warp's
        __syncthreads();
        cells = s_cells;
    } else {
        st = team_rows_static<S, W, 32 * W>(a, s_part, &s_fail, cells);
        if (st == ST_OK) team_fill_static<W, WIDE>(a, tsm);
    }
    if (st != ST_OK) {
        if (threadIdx.x == 0) {
            a.out[0] = st;
            a.out[1] = 0;
            a.out[2] = 0;
            a.out[3] = 0;
        }
        return;
    }
    if (threadIdx.x < 32) team_finish<WIDE, 8>(a, tsm, S::BYTES, cells, threadIdx.x);
}

}  // namespace pb

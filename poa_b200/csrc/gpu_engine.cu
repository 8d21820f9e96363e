// gpu_engine.cu - host side of the plain DP path (see gpu_engine.h).
#include "gpu_engine.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <stdexcept>

#include "team.cuh"

namespace pb {

void cuda_check(int err, const char* what) {
    if (err != cudaSuccess)
        throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString((cudaError_t)err));
}

namespace {

inline size_t up16(size_t x) { return (x + 15) & ~(size_t)15; }

// Row-store blocks of a job (exact for the static band, the worst case for the
// adaptive band) and the columns of its widest row.
void job_capacity(const HostWindow& w, int qlen, bool adaptive, int f, int wband, int64_t& blocks, int& cols) {
    const int m = qlen + 1;
    blocks = 0;
    cols = 8;
    if (adaptive) {
        // a row starts near 2 * wband columns and widens with the band state, up to the
        // whole query; rows beyond the team's columns take more laps
        blocks = (int64_t)w.n * (m / BLK + 1);
        cols = (int)std::min<int64_t>((int64_t)(m / BLK + 1) * BLK, 6 * (int64_t)wband + STRIP);
        return;
    }
    for (int i = 0; i < w.n; i++) {
        int Bs, Be;
        band_static(f, w.hq[i], w.tq[i], m, wband, Bs, Be);
        if (i == 0) Bs = 0;
        const int bn = std::max(0, Be - Bs - 1);
        blocks += bn;
        cols = std::max(cols, ((Be - 2) / SBLK - Bs / SBLK + 1) * STRIP);
    }
}

// A row's predecessor records in the backtrack's priority order (in_weight
// descending, in-list position ascending; src/align.cpp:1601, 1637, 1708 keep
// the first maximum), see TeamJob::ed.
void pack_edges(const HostWindow& w, int4* ed) {
    for (int r = 0; r < w.n; r++) {
        const int e0 = w.in_ptr[r], d = w.in_ptr[r + 1] - e0;
        int order[8];
        std::vector<int> big;
        int* o = order;
        if (d > 8) {
            big.resize(d);
            o = big.data();
        }
        for (int k = 0; k < d; k++) {
            int at = k;
            while (at > 0 && w.in_w[e0 + o[at - 1]] < w.in_w[e0 + k]) {
                o[at] = o[at - 1];
                at--;
            }
            o[at] = k;
        }
        const int least = w.ind[r] / 10;
        for (int k = 0; k < d; k++) {
            const int e = e0 + o[k];
            ed[e0 + k] = make_int4((w.in_row[e] << 4) | (w.in_w[e] >= least ? 8 : 0) | w.in_base[e], 0, 0, 0);
        }
    }
}

template <int W, bool ADAPT, bool WIDE>
void launch_team(int njobs, const TeamJob* d_jobs, cudaStream_t s) {
    typedef TeamSmem<W, ADAPT, WIDE> S;
    cuda_check(cudaFuncSetAttribute(k_align<W, ADAPT, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES),
               "smem attr (k_align)");
    k_align<W, ADAPT, WIDE><<<njobs, S::THREADS, S::BYTES, s>>>(d_jobs);
}

// One warp per 128 columns of the widest row, up to 16 (rows beyond that take
// laps, with every predecessor from the row store). Measured against the record
// fill, which took 4,096 columns at a time: three static reads of 45 kb 298 -> 210
// ms, of 60 kb 552 -> 294; full band, reads of 2.5 kb 46 -> 32, of 5 kb 110 -> 60;
// wide cells, full band, 1.2 kb 12.7 -> 6.2, 2.5 kb 36.1 -> 33.2 (39.5 with 8 warps at
// most), 5 kb 109 -> 77; static wide, 30 kb 164 -> 80.
void launch_teams(bool adaptive, bool wide, int cols, int njobs, const TeamJob* d, cudaStream_t s) {
    const int strips = (cols + STRIP - 1) / STRIP;
    if (wide && adaptive) {
        launch_team<8, true, true>(njobs, d, s);
    } else if (wide) {
        // (8 bytes a cell: 16 warps keep 8 rows in shared memory, 8 or 12 warps 16)
        if (strips <= 8) launch_team<8, false, true>(njobs, d, s);
        else if (strips <= 12) launch_team<12, false, true>(njobs, d, s);
        else launch_team<16, false, true>(njobs, d, s);
    } else if (adaptive) {
        if (strips <= 2) launch_team<2, true, false>(njobs, d, s);
        else if (strips <= 4) launch_team<4, true, false>(njobs, d, s);
        else if (strips <= 8) launch_team<8, true, false>(njobs, d, s);
        else if (strips <= 12) launch_team<12, true, false>(njobs, d, s);
        else launch_team<16, true, false>(njobs, d, s);
    } else {
        if (strips <= 2) launch_team<2, false, false>(njobs, d, s);
        else if (strips <= 3) launch_team<3, false, false>(njobs, d, s);
        else if (strips <= 4) launch_team<4, false, false>(njobs, d, s);
        else if (strips <= 6) launch_team<6, false, false>(njobs, d, s);
        else if (strips <= 8) launch_team<8, false, false>(njobs, d, s);
        else if (strips <= 10) launch_team<10, false, false>(njobs, d, s);
        else if (strips <= 12) launch_team<12, false, false>(njobs, d, s);
        else launch_team<16, false, false>(njobs, d, s);
    }
}

}  // namespace

GpuEngine::GpuEngine(int device) : device_(device) {
    cuda_check(cudaSetDevice(device), "cudaSetDevice");
    cudaStream_t s;
    cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "cudaStreamCreate");
    stream_ = s;
    cudaEvent_t e0, e1;
    cuda_check(cudaEventCreate(&e0), "cudaEventCreate");
    cuda_check(cudaEventCreate(&e1), "cudaEventCreate");
    ev0_ = e0;
    ev1_ = e1;
}

GpuEngine::~GpuEngine() {
    cudaSetDevice(device_);
    if (dbuf_) cudaFree(dbuf_);
    if (hbuf_) cudaFreeHost(hbuf_);
    if (ev0_) cudaEventDestroy((cudaEvent_t)ev0_);
    if (ev1_) cudaEventDestroy((cudaEvent_t)ev1_);
    if (stream_) cudaStreamDestroy((cudaStream_t)stream_);
}

void GpuEngine::reserve_device(size_t bytes) {
    if (bytes <= dcap_) return;
    size_t cap = std::max(bytes, dcap_ * 2);
    if (dbuf_) cuda_check(cudaFree(dbuf_), "cudaFree");
    dbuf_ = nullptr;
    dcap_ = 0;
    cuda_check(cudaMalloc((void**)&dbuf_, cap), "cudaMalloc(arena)");
    dcap_ = cap;
}

void GpuEngine::reserve_host(size_t bytes) {
    if (bytes <= hcap_) return;
    size_t cap = std::max(bytes, hcap_ * 2);
    if (hbuf_) cuda_check(cudaFreeHost(hbuf_), "cudaFreeHost");
    hbuf_ = nullptr;
    hcap_ = 0;
    cuda_check(cudaMallocHost((void**)&hbuf_, cap), "cudaMallocHost(staging)");
    hcap_ = cap;
}

void GpuEngine::align_many(const std::vector<const HostWindow*>& wins, const std::vector<const uint8_t*>& qs,
                           const std::vector<int32_t>& qlens, const std::vector<int32_t>& abs, const Params& p,
                           std::vector<AlignOut>& outs) {
    const int J = (int)wins.size();
    outs.assign(J, AlignOut());
    if (J == 0) return;
    // one launch runs one kind of band
    bool any_adaptive = false, any_static = false;
    for (int t = 0; t < J; t++) (p.f > 0 && abs[t] ? any_adaptive : any_static) = true;
    if (any_adaptive && any_static) throw std::invalid_argument("align_many: one kind of band a call");
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    cudaStream_t s = (cudaStream_t)stream_;
    const Scoring sc = scoring_of(p);

    struct Lay {
        size_t in_ptr, ed, hq, tq, ra, out_row, qs;
        size_t rowi, fr, fe, state, store, res;
        int64_t blocks;
        int32_t moves_cap;
        int w;
    };
    std::vector<Lay> L(J);
    size_t up = up16(sizeof(TeamJob) * J);
    int cols = 8;
    bool wide = false;
    for (int t = 0; t < J; t++) {
        const HostWindow& w = *wins[t];
        const size_t n = (size_t)w.n, E = w.in_row.size();
        Lay& l = L[t];
        const int m = qlens[t] + 1;
        l.w = p.b + (p.f ? m / p.f : 0);
        l.in_ptr = up; up += up16(4 * (n + 1));
        l.ed = up; up += up16(16 * E);
        l.hq = l.tq = l.ra = l.out_row = up;
        if (any_adaptive) {
            l.ra = up; up += up16(32 * n);
            l.out_row = up; up += up16(4 * E);
        } else {
            l.hq = up; up += up16(4 * n);
            l.tq = up; up += up16(4 * n);
        }
        l.qs = up; up += up16((size_t)qs_bytes(qlens[t]));
        int c;
        job_capacity(w, qlens[t], any_adaptive, p.f, l.w, l.blocks, c);
        cols = std::max(cols, c);
        wide = wide || !cell_packable(sc, w.n, m);
        l.moves_cap = w.n + m + 8;
    }
    size_t res_begin = up;
    size_t pos = up;
    for (int t = 0; t < J; t++) {
        L[t].res = pos;
        pos += up16(16 + 4 * (size_t)L[t].moves_cap);
    }
    size_t res_end = pos;
    for (int t = 0; t < J; t++) {
        const size_t n = (size_t)wins[t]->n;
        L[t].rowi = pos; pos += 16 * n;
        L[t].fr = pos; pos += any_adaptive ? 0 : 16 * n;
        L[t].fe = pos; pos += 16 * wins[t]->in_row.size();
        L[t].state = pos; pos += any_adaptive ? 32 * n : 0;
        L[t].store = pos; pos += up16((size_t)L[t].blocks * BLK * (wide ? 8 : 4));
    }
    reserve_device(pos);
    reserve_host(res_end);

    char* h = hbuf_;
    char* d = dbuf_;
    TeamJob* jobs = reinterpret_cast<TeamJob*>(h);
    for (int t = 0; t < J; t++) {
        const HostWindow& w = *wins[t];
        const Lay& l = L[t];
        std::memcpy(h + l.in_ptr, w.in_ptr.data(), 4 * (size_t)(w.n + 1));
        pack_edges(w, reinterpret_cast<int4*>(h + l.ed));
        if (any_adaptive) {
            int4* ra = reinterpret_cast<int4*>(h + l.ra);
            for (int r = 0; r < w.n; r++) {
                ra[2 * r] = make_int4(w.in_ptr[r], w.out_ptr[r], w.hq[r], w.tq[r]);
                ra[2 * r + 1] = make_int4(w.hq_loc[r], w.base[r], w.in_ptr[r + 1] - w.in_ptr[r],
                                          w.out_ptr[r + 1] - w.out_ptr[r]);
            }
            std::memcpy(h + l.out_row, w.out_row.data(), 4 * w.out_row.size());
        } else {
            std::memcpy(h + l.hq, w.hq.data(), 4 * (size_t)w.n);
            std::memcpy(h + l.tq, w.tq.data(), 4 * (size_t)w.n);
        }
        make_qs(qs[t], qlens[t], reinterpret_cast<uint8_t*>(h + l.qs));
        TeamJob a;
        std::memset(&a, 0, sizeof(a));
        a.n = w.n;
        a.qlen = qlens[t];
        a.f = p.f;
        a.w = l.w;
        a.k = cell_consts(sc);
        a.in_ptr = reinterpret_cast<const int32_t*>(d + l.in_ptr);
        a.ed = reinterpret_cast<int4*>(d + l.ed);
        a.hq = reinterpret_cast<const int32_t*>(d + l.hq);
        a.tq = reinterpret_cast<const int32_t*>(d + l.tq);
        a.ra = reinterpret_cast<const int4*>(d + l.ra);
        a.out_row = reinterpret_cast<const int32_t*>(d + l.out_row);
        a.qs = reinterpret_cast<const uint8_t*>(d + l.qs);
        a.rowi = reinterpret_cast<int4*>(d + l.rowi);
        a.fr = reinterpret_cast<int4*>(d + l.fr);
        a.fe = reinterpret_cast<int4*>(d + l.fe);
        a.state = reinterpret_cast<int32_t*>(d + l.state);
        a.store = d + l.store;
        a.store_cap = l.blocks;
        a.out = reinterpret_cast<int32_t*>(d + l.res);
        a.moves = reinterpret_cast<int32_t*>(d + l.res + 16);
        a.moves_cap = l.moves_cap;
        jobs[t] = a;
    }
    cuda_check(cudaMemcpyAsync(d, h, res_begin, cudaMemcpyHostToDevice, s), "cudaMemcpyAsync(H2D)");
    if (timing) cuda_check(cudaEventRecord((cudaEvent_t)ev0_, s), "cudaEventRecord");
    launch_teams(any_adaptive, wide, cols, J, reinterpret_cast<const TeamJob*>(d), s);
    cuda_check(cudaGetLastError(), "k_align launch");
    if (timing) cuda_check(cudaEventRecord((cudaEvent_t)ev1_, s), "cudaEventRecord");
    cuda_check(cudaMemcpyAsync(h + res_begin, d + res_begin, res_end - res_begin, cudaMemcpyDeviceToHost, s),
               "cudaMemcpyAsync(D2H)");
    cuda_check(cudaStreamSynchronize(s), "DP kernel");
    stats.launches++;
    stats.alignments += J;
    stats.h2d_bytes += (int64_t)res_begin;
    stats.d2h_bytes += (int64_t)(res_end - res_begin);
    if (timing) {
        float ms = 0.f;
        cuda_check(cudaEventElapsedTime(&ms, (cudaEvent_t)ev0_, (cudaEvent_t)ev1_), "cudaEventElapsedTime");
        stats.kernel_ms += ms;
    }
    for (int t = 0; t < J; t++) {
        const int32_t* o = reinterpret_cast<const int32_t*>(h + L[t].res);
        AlignOut& r = outs[t];
        r.status = o[0];
        r.score = o[1];
        r.cells = o[3];
        stats.cells += o[3];
        if (r.status == ST_OK) {
            int nm = std::min(o[2], L[t].moves_cap);
            r.moves.assign(o + 4, o + 4 + nm);
        }
    }
}

}  // namespace pb

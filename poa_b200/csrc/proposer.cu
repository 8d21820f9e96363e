// proposer.cu - features, network (training and inference) and window plan of
// the learned band proposer; see proposer.h for what it predicts and why.
//
// Everything here is hand-written CUDA: the network kernel (prop_net.cuh),
// Adam, the minimizer feature kernel and the plan kernel.
#include "proposer.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>
#include <stdexcept>

#include "batch.h"
#include "gpu_engine.h"
#include "prop_net.cuh"
#include "sketch.h"

namespace pb {
namespace {

typedef __nv_bfloat16 bf16;

constexpr int T = PROP_BINS;
using net::OB5;
using net::OW1;
using net::OW2;
using net::OW3;
using net::OW4;
using net::OW5;
constexpr int KC1 = net::KC1, KC = net::KC;
// extras
constexpr int X_MEAN = 0, X_STD = 4, X_NODE_MARGIN = 8, X_TB_MARGIN = 9, X_SPILL_PER_ROW = 10, X_SPILL_MIN = 11;

inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

// ---------------------------------------------------------------------------
// elementwise kernels (grid-stride)
#define GRID_STRIDE(i, n) for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

inline unsigned grid_of(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(n, 256), 148 * 16)); }

__global__ void k_to_bf16(const float* __restrict__ x, bf16* __restrict__ y, int64_t n) {
    GRID_STRIDE(i, n) y[i] = __float2bfloat16(x[i]);
}

// Adam on the FP32 master weights, refreshing the BF16 copy
__global__ void k_adam(float* __restrict__ w, bf16* __restrict__ wb, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    GRID_STRIDE(i, n) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        wb[i] = __float2bfloat16(wi);
    }
}

// ---------------------------------------------------------------------------
// minimizer features: one CTA per window, a hash table per CTA in global memory
constexpr int FT_THREADS = 128;
constexpr int FT_TILE = 1024;      // k-mer end positions per tile
constexpr int FT_MAXW = 32;        // largest minimizer window supported
constexpr int FT_MAXK = 28;

__device__ __forceinline__ int nt4_dev2(uint8_t c) {
    switch (c | 0x20) {
        case 'a': return 0;
        case 'c': return 1;
        case 'g': return 2;
        case 't': return 3;
        default: return 4;
    }
}

__device__ __forceinline__ uint32_t mm_key(uint64_t h) {
    const uint32_t k = (uint32_t)(h ^ (h >> 32));
    return k ? k : 1u;
}

// For the tile [p0, p0 + FT_TILE) of a read: hashes of k-mers ending at
// p0 - (w-1) .. p0 + FT_TILE + w - 2 (UINT64_MAX where no valid k-mer ends),
// then a flag per tile position: the k-mer ending there is the minimum of a
// full window of w consecutive valid k-mers (src/minimizer.cpp:60-135 for
// reads without an ambiguous base; equal minima in a window are all kept).
__device__ void sketch_tile(const uint8_t* rd, int len, int p0, int k, int w, uint8_t* sb, uint64_t* sh, uint8_t* flag) {
    const int H = FT_TILE + 2 * (w - 1);
    const int q0 = p0 - (w - 1) - (k - 1);  // first base needed
    const int nb = H + k - 1;
    for (int i = threadIdx.x; i < nb; i += FT_THREADS) {
        const int q = q0 + i;
        sb[i] = (q >= 0 && q < len) ? (uint8_t)nt4_dev2(rd[q]) : 4;
    }
    __syncthreads();
    const uint64_t mask = (k >= 32) ? ~0ull : ((1ull << (2 * k)) - 1);
    for (int i = threadIdx.x; i < H; i += FT_THREADS) {
        const int p = p0 - (w - 1) + i;  // k-mer end position
        uint64_t h = UINT64_MAX;
        if (p >= k - 1 && p < len) {
            uint64_t code = 0;
            bool ok = true;
            for (int j = 0; j < k; j++) {
                const int c = sb[i + j];
                ok &= c < 4;
                code = (code << 2) | (uint64_t)(c & 3);
            }
            if (ok) h = hash64(code & mask, mask);
        }
        sh[i] = h;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < FT_TILE; i += FT_THREADS) {
        const int c = i + (w - 1);  // index of the tile position in sh
        const uint64_t hp = sh[c];
        bool mn = false;
        if (hp != UINT64_MAX) {
            for (int s = c - (w - 1); s <= c && !mn; s++) {
                uint64_t wm = UINT64_MAX;
                bool full = true;
                for (int j = s; j < s + w; j++) {
                    full &= sh[j] != UINT64_MAX;
                    wm = sh[j] < wm ? sh[j] : wm;
                }
                mn = full && wm == hp;
            }
        }
        flag[i] = mn;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(FT_THREADS) k_features(const uint8_t* __restrict__ seq, const int64_t* __restrict__ read_off,
                                                        const int32_t* __restrict__ read_len,
                                                        const int32_t* __restrict__ win_off, int n_windows, int k, int w,
                                                        unsigned long long* __restrict__ tabs, int tab_bits,
                                                        float* __restrict__ X) {
    __shared__ uint8_t sb[FT_TILE + 2 * FT_MAXW + FT_MAXK];
    __shared__ uint64_t sh[FT_TILE + 2 * FT_MAXW];
    __shared__ uint8_t flag[FT_TILE];
    __shared__ float acc[T][3];
    const int tsize = 1 << tab_bits;
    unsigned long long* tab = tabs + (size_t)blockIdx.x * tsize;
    for (int win = blockIdx.x; win < n_windows; win += gridDim.x) {
        for (int i = threadIdx.x; i < tsize; i += FT_THREADS) tab[i] = 0ull;
        __syncthreads();
        const int r0 = win_off[win], r1 = win_off[win + 1];
        const int R = r1 - r0;
        // pass 1: count every minimizer of every read
        for (int r = r0; r < r1; r++) {
            const uint8_t* rd = seq + read_off[r];
            const int len = read_len[r];
            for (int p0 = 0; p0 < len; p0 += FT_TILE) {
                sketch_tile(rd, len, p0, k, w, sb, sh, flag);
                for (int i = threadIdx.x; i < FT_TILE; i += FT_THREADS) {
                    if (!flag[i]) continue;
                    const uint32_t key = mm_key(sh[i + w - 1]);
                    uint32_t slot = (key * 2654435761u) >> (32 - tab_bits);
                    for (int probe = 0; probe < tsize; probe++) {  // bounded: at most one pass over the table
                        unsigned long long cur = tab[slot];
                        if (cur == 0ull) {
                            cur = atomicCAS(&tab[slot], 0ull, ((unsigned long long)key << 32) | 1ull);
                            if (cur == 0ull) break;
                        }
                        if ((uint32_t)(cur >> 32) == key) {
                            atomicAdd(&tab[slot], 1ull);
                            break;
                        }
                        slot = (slot + 1) & (uint32_t)(tsize - 1);
                    }
                }
                __syncthreads();
            }
        }
        __syncthreads();
        // pass 2: per read and bin, density / anchored fraction / multiplicity
        const int L0 = R > 0 ? read_len[r0] : 0;
        for (int r = r0; r < r1; r++) {
            const uint8_t* rd = seq + read_off[r];
            const int len = read_len[r];
            for (int i = threadIdx.x; i < T * 3; i += FT_THREADS) (&acc[0][0])[i] = 0.f;
            __syncthreads();
            for (int p0 = 0; p0 < len; p0 += FT_TILE) {
                sketch_tile(rd, len, p0, k, w, sb, sh, flag);
                for (int i = threadIdx.x; i < FT_TILE; i += FT_THREADS) {
                    if (!flag[i]) continue;
                    const uint32_t key = mm_key(sh[i + w - 1]);
                    uint32_t slot = (key * 2654435761u) >> (32 - tab_bits);
                    int cnt = 0;
                    for (int probe = 0; probe < tsize; probe++) {
                        const unsigned long long cur = tab[slot];
                        if (cur == 0ull) break;
                        if ((uint32_t)(cur >> 32) == key) {
                            cnt = (int)(cur & 0xffffffffu);
                            break;
                        }
                        slot = (slot + 1) & (uint32_t)(tsize - 1);
                    }
                    const int others = max(cnt - 1, 0);
                    const int bin = (int)((int64_t)(p0 + i) * T / max(len, 1));
                    atomicAdd(&acc[bin][0], 1.f);
                    atomicAdd(&acc[bin][1], others > 0 ? 1.f : 0.f);
                    atomicAdd(&acc[bin][2], (float)min(others, max(R - 1, 1)));
                }
                __syncthreads();
            }
            for (int b = threadIdx.x; b < T; b += FT_THREADS) {
                const float blen = fmaxf((float)len / T, 1.f);
                const float nm = acc[b][0];
                float* x = X + ((int64_t)r * T + b) * PROP_CIN;
                x[0] = nm * (float)(w + 1) / (2.f * blen);
                x[1] = nm > 0.f ? acc[b][1] / nm : 0.f;
                x[2] = nm > 0.f ? 10.f * acc[b][2] / (nm * (float)max(R - 1, 1)) : 0.f;
                x[3] = (float)len / 2048.f;
                x[4] = (float)L0 / 2048.f;
                x[5] = (float)(r - r0) / 100.f;
                x[6] = (float)R / 100.f;
                x[7] = ((float)b + 0.5f) / T;
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// per-window plan from the per-read predictions (one thread per window)
__global__ void k_plan(const float* __restrict__ pred, const int32_t* __restrict__ read_len,
                       const int32_t* __restrict__ win_off, int n_windows, const float* __restrict__ extra,
                       int32_t* __restrict__ nodes_out, int64_t* __restrict__ tb_out, int64_t* __restrict__ spill_out,
                       float* __restrict__ cost_out, int64_t* __restrict__ cells_out) {
    GRID_STRIDE(wi, n_windows) {
        const int w = (int)wi;
        const int r0 = win_off[w], r1 = win_off[w + 1];
        double nodes = r1 > r0 ? 2.0 + read_len[r0] : 2.0;
        double maxtb = 0.0, maxcells = 0.0, maxrows = 0.0, cost = 0.0;
        for (int r = r0 + 1; r < r1; r++) {
            const float* y = pred + (int64_t)r * PROP_OUT;
            const double rows = nodes;
            const double m = (double)read_len[r] + 1.0;
            const double cells = fmin(fmax((double)y[1], 0.01), 1.0) * rows * m;
            const double bpc = fmin(fmax((double)y[2], 1.0), 4.0);
            maxtb = fmax(maxtb, cells * bpc);
            maxcells = fmax(maxcells, cells);
            maxrows = fmax(maxrows, rows);
            cost += cells;
            nodes += fmax((double)y[0], 0.0) * read_len[r];
        }
        nodes_out[w] = (int32_t)fmin(nodes * extra[X_NODE_MARGIN] + 64.0, 2.0e9);
        tb_out[w] = (int64_t)(maxtb * extra[X_TB_MARGIN]) + 4096;
        spill_out[w] = (int64_t)fmax((double)extra[X_SPILL_MIN], maxrows * extra[X_SPILL_PER_ROW]);
        cost_out[w] = (float)cost;
        cells_out[w] = (int64_t)(maxcells * extra[X_TB_MARGIN]) + 4096;
    }
}

}  // namespace

Proposer::Proposer(int device) : device_(device) {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    host_w_.assign(PROP_NWEIGHTS, 0.f);
    cuda_check(cudaMalloc(&d_w_, 4 * (size_t)PROP_NPARAM), "cudaMalloc(proposer)");
    cuda_check(cudaMalloc(&d_wb_, 2 * (size_t)PROP_NPARAM), "cudaMalloc(proposer)");
    cuda_check(cudaMalloc(&d_g_, 4 * (size_t)(PROP_NPARAM + 1)), "cudaMalloc(proposer)");
    cuda_check(cudaMalloc(&d_m_, 4 * (size_t)PROP_NPARAM), "cudaMalloc(proposer)");
    cuda_check(cudaMalloc(&d_v_, 4 * (size_t)PROP_NPARAM), "cudaMalloc(proposer)");
    cuda_check(cudaMalloc(&d_extra_, 4 * (size_t)PROP_NEXTRA), "cudaMalloc(proposer)");
    // default initialisation: He-uniform weights from a fixed seed, zero biases,
    // identity standardisation, unit margins
    std::mt19937_64 rng(12345);
    auto init = [&](int off, int fan_out, int fan_in) {
        const float lim = std::sqrt(6.f / (float)fan_in);
        std::uniform_real_distribution<float> u(-lim, lim);
        for (int i = 0; i < fan_out * fan_in; i++) host_w_[off + i] = u(rng);
    };
    init(OW1, PROP_CH, KC1);
    init(OW2, PROP_CH, KC);
    init(OW3, PROP_CH, KC);
    init(OW4, PROP_CH, PROP_CH);
    init(OW5, PROP_OUT, PROP_CH);
    for (int k = 0; k < PROP_OUT; k++) host_w_[PROP_NPARAM + X_STD + k] = 1.f;
    host_w_[PROP_NPARAM + X_NODE_MARGIN] = 1.f;
    host_w_[PROP_NPARAM + X_TB_MARGIN] = 1.f;
    host_w_[PROP_NPARAM + X_SPILL_PER_ROW] = 8.f;
    host_w_[PROP_NPARAM + X_SPILL_MIN] = 65536.f;
    set_weights(host_w_.data());
}

Proposer::~Proposer() {
    cudaSetDevice(device_);
    if (graph_exec_) cudaGraphExecDestroy((cudaGraphExec_t)graph_exec_);
    for (void* p : {(void*)d_w_, (void*)d_wb_, (void*)d_g_, (void*)d_m_, (void*)d_v_, (void*)d_extra_, (void*)d_part_, d_io_, d_tab_,
                    d_plan_, (void*)d_feat_, (void*)d_pred_})
        if (p) cudaFree(p);
}

void Proposer::upload_bf16(void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    k_to_bf16<<<grid_of(PROP_NPARAM), 256, 0, s>>>(d_w_, (bf16*)d_wb_, PROP_NPARAM);
    cuda_check(cudaGetLastError(), "k_to_bf16");
}

void Proposer::set_weights(const float* w) {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    std::memcpy(host_w_.data(), w, 4 * (size_t)PROP_NWEIGHTS);
    for (int k = 0; k < PROP_OUT; k++)
        if (!(host_w_[PROP_NPARAM + X_STD + k] > 0.f)) throw std::invalid_argument("proposer: output std must be > 0");
    cuda_check(cudaMemcpy(d_w_, host_w_.data(), 4 * (size_t)PROP_NPARAM, cudaMemcpyHostToDevice), "H2D weights");
    cuda_check(cudaMemcpy(d_extra_, host_w_.data() + PROP_NPARAM, 4 * (size_t)PROP_NEXTRA, cudaMemcpyHostToDevice),
               "H2D extras");
    cuda_check(cudaMemset(d_m_, 0, 4 * (size_t)PROP_NPARAM), "memset");
    cuda_check(cudaMemset(d_v_, 0, 4 * (size_t)PROP_NPARAM), "memset");
    upload_bf16(nullptr);
    cuda_check(cudaDeviceSynchronize(), "set_weights");
}

void Proposer::get_weights(float* w) const {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    std::vector<float> h(PROP_NPARAM);
    cuda_check(cudaMemcpy(h.data(), d_w_, 4 * (size_t)PROP_NPARAM, cudaMemcpyDeviceToHost), "D2H weights");
    std::memcpy(w, h.data(), 4 * (size_t)PROP_NPARAM);
    std::memcpy(w + PROP_NPARAM, host_w_.data() + PROP_NPARAM, 4 * (size_t)PROP_NEXTRA);
}

void* Proposer::io(size_t bytes) {
    if (bytes > io_bytes_) {
        if (d_io_) cuda_check(cudaFree(d_io_), "cudaFree");
        d_io_ = nullptr;
        io_bytes_ = 0;
        cuda_check(cudaMalloc(&d_io_, bytes), "cudaMalloc(proposer batch)");
        io_bytes_ = bytes;
    }
    return d_io_;
}

// CTAs of the network kernel for n reads: one per SM at most (a CTA holds the
// weights and a tile in most of an SM's shared memory), persistent over tiles
int Proposer::net_grid(int64_t n) const {
    int sms = 0;
    cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_), "attr");
    return (int)std::min<int64_t>(cdiv(n, net::RT), sms);
}

// Loss (added to the word after the gradient) and gradient of reads idx[0 .. n)
// of device arrays X, Y into d_g_.
void Proposer::loss_and_gradient(const float* X, const float* Y, const int32_t* idx, int64_t n, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const int grid = net_grid(n);
    if (grid > part_ctas_) {
        if (d_part_) cuda_check(cudaFree(d_part_), "cudaFree");
        d_part_ = nullptr;
        part_ctas_ = 0;
        cuda_check(cudaMalloc(&d_part_, 4 * (size_t)net::PART * grid), "cudaMalloc(proposer sums)");
        part_ctas_ = grid;
    }
    cuda_check(cudaFuncSetAttribute(net::k_net<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(net::Smem)),
               "smem attr (k_net)");
    net::k_net<true><<<grid, net::THREADS, sizeof(net::Smem), s>>>(X, Y, idx, n, (const bf16*)d_wb_, d_w_, d_extra_, nullptr,
                                                                  d_part_);
    net::k_net_sum<<<(unsigned)cdiv(PROP_NPARAM + 1, 128), 128, 0, s>>>(d_part_, grid, d_g_, d_g_ + PROP_NPARAM);
    cuda_check(cudaGetLastError(), "proposer gradient");
}

float Proposer::train(const float* X, const float* Y, int64_t n, int epochs, int batch, float lr, uint64_t seed,
                      float* losses) {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    if (n <= 0 || batch <= 0 || epochs <= 0) throw std::invalid_argument("proposer: empty training set");
    // standardisation of the targets from the training set
    for (int k = 0; k < PROP_OUT; k++) {
        double s = 0.0, s2 = 0.0;
        for (int64_t i = 0; i < n; i++) {
            s += Y[i * PROP_OUT + k];
            s2 += (double)Y[i * PROP_OUT + k] * Y[i * PROP_OUT + k];
        }
        const double mean = s / n, var = std::max(s2 / n - mean * mean, 1e-12);
        host_w_[PROP_NPARAM + X_MEAN + k] = (float)mean;
        host_w_[PROP_NPARAM + X_STD + k] = (float)std::sqrt(var);
    }
    cuda_check(cudaMemcpy(d_extra_, host_w_.data() + PROP_NPARAM, 4 * (size_t)PROP_NEXTRA, cudaMemcpyHostToDevice),
               "H2D extras");
    cudaStream_t s = nullptr;
    float *dX = nullptr, *dY = nullptr;
    int32_t* dIdx = nullptr;
    cuda_check(cudaMalloc(&dX, 4 * (size_t)n * T * PROP_CIN), "cudaMalloc(train X)");
    cuda_check(cudaMalloc(&dY, 4 * (size_t)n * PROP_OUT), "cudaMalloc(train Y)");
    cuda_check(cudaMalloc(&dIdx, 4 * (size_t)n), "cudaMalloc(train idx)");
    cuda_check(cudaMemcpy(dX, X, 4 * (size_t)n * T * PROP_CIN, cudaMemcpyHostToDevice), "H2D X");
    cuda_check(cudaMemcpy(dY, Y, 4 * (size_t)n * PROP_OUT, cudaMemcpyHostToDevice), "H2D Y");
    std::vector<int32_t> idx(n);
    std::iota(idx.begin(), idx.end(), 0);
    std::mt19937_64 rng(seed);
    int step = 0;
    float last = 0.f;
    for (int ep = 0; ep < epochs; ep++) {
        std::shuffle(idx.begin(), idx.end(), rng);
        cuda_check(cudaMemcpy(dIdx, idx.data(), 4 * (size_t)n, cudaMemcpyHostToDevice), "H2D idx");
        cuda_check(cudaMemset(d_g_ + PROP_NPARAM, 0, 4), "memset loss");
        int nbatches = 0;
        for (int64_t b0 = 0; b0 < n; b0 += batch) {
            const int64_t nb = std::min<int64_t>(batch, n - b0);
            loss_and_gradient(dX, dY, dIdx + b0, nb, s);
            step++;
            const float b1 = 0.9f, b2 = 0.999f;
            k_adam<<<grid_of(PROP_NPARAM), 256, 0, s>>>(d_w_, (bf16*)d_wb_, d_g_, d_m_, d_v_, PROP_NPARAM, lr, b1, b2,
                                                        1e-8f, 1.f - std::pow(b1, (float)step),
                                                        1.f - std::pow(b2, (float)step));
            cuda_check(cudaGetLastError(), "proposer train step");
            nbatches++;
        }
        float lsum = 0.f;
        cuda_check(cudaMemcpy(&lsum, d_g_ + PROP_NPARAM, 4, cudaMemcpyDeviceToHost), "D2H loss");
        last = lsum / (float)std::max(nbatches, 1);
        if (losses) losses[ep] = last;
    }
    cudaFree(dX);
    cudaFree(dY);
    cudaFree(dIdx);
    return last;
}

float Proposer::gradient(const float* X, const float* Y, int64_t n, float* grad) {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    if (n <= 0 || n > 4096) throw std::invalid_argument("proposer: gradient batch must hold 1..4096 reads");
    const size_t xb = up256(4 * (size_t)n * T * PROP_CIN);
    float* dX = (float*)io(xb + 4 * (size_t)n * PROP_OUT);
    float* dY = (float*)((char*)dX + xb);
    cuda_check(cudaMemcpy(dX, X, 4 * (size_t)n * T * PROP_CIN, cudaMemcpyHostToDevice), "H2D X");
    cuda_check(cudaMemcpy(dY, Y, 4 * (size_t)n * PROP_OUT, cudaMemcpyHostToDevice), "H2D Y");
    cuda_check(cudaMemsetAsync(d_g_ + PROP_NPARAM, 0, 4, nullptr), "memset loss");
    loss_and_gradient(dX, dY, nullptr, n, nullptr);
    std::vector<float> h(PROP_NPARAM + 1);
    cuda_check(cudaMemcpy(h.data(), d_g_, 4 * (size_t)(PROP_NPARAM + 1), cudaMemcpyDeviceToHost), "D2H grad");
    std::memcpy(grad, h.data(), 4 * (size_t)PROP_NPARAM);
    return h[PROP_NPARAM];
}

void Proposer::predict_device(const float* dX, int64_t n, float* dY, void* stream) {
    if (n <= 0) return;
    cuda_check(cudaFuncSetAttribute(net::k_net<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(net::Smem)),
               "smem attr (k_net)");
    net::k_net<false><<<net_grid(n), net::THREADS, sizeof(net::Smem), (cudaStream_t)stream>>>(
        dX, nullptr, nullptr, n, (const bf16*)d_wb_, d_w_, d_extra_, dY, nullptr);
    cuda_check(cudaGetLastError(), "proposer predict");
}

// Host arrays go through the object's device buffer a chunk at a time (16 K
// reads, 16 MiB), so it stays small whatever the call.
constexpr int64_t PREDICT_CHUNK = 16384;

void Proposer::predict_host(const float* X, int64_t n, float* Y) {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    const int64_t cap = std::min<int64_t>(std::max<int64_t>(n, 1), PREDICT_CHUNK);
    const size_t xb = up256(4 * (size_t)cap * T * PROP_CIN);
    float* dX = (float*)io(xb + 4 * (size_t)cap * PROP_OUT);
    float* dY = (float*)((char*)dX + xb);
    for (int64_t b0 = 0; b0 < n; b0 += cap) {
        const int64_t nb = std::min<int64_t>(cap, n - b0);
        cuda_check(cudaMemcpy(dX, X + b0 * T * PROP_CIN, 4 * (size_t)nb * T * PROP_CIN, cudaMemcpyHostToDevice), "H2D X");
        predict_device(dX, nb, dY, nullptr);
        cuda_check(cudaMemcpy(Y + b0 * PROP_OUT, dY, 4 * (size_t)nb * PROP_OUT, cudaMemcpyDeviceToHost), "D2H Y");
    }
}

void Proposer::features(const DeviceWindows& dw, int k, int w, float* dX, void* stream) {
    if (dw.n_windows <= 0) return;
    int bits = 0, grid = 0;
    features_prep(dw, k, w, bits, grid);
    features_launch(dw, k, w, bits, grid, dX, stream);
}

void Proposer::features_launch(const DeviceWindows& dw, int k, int w, int bits, int grid, float* dX, void* stream) {
    k_features<<<grid, FT_THREADS, 0, (cudaStream_t)stream>>>(dw.seq, dw.read_off, dw.read_len, dw.win_off,
                                                               dw.n_windows, k, w, (unsigned long long*)d_tab_, bits,
                                                               dX);
    cuda_check(cudaGetLastError(), "k_features");
}

// hash-table size and grid of the feature kernel; allocates its scratch
void Proposer::features_prep(const DeviceWindows& dw, int k, int w, int& bits_out, int& grid_out) {
    if (k < 1 || k > FT_MAXK || w < 1 || w > FT_MAXW) throw std::invalid_argument("proposer: k or w out of range");
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    // table: at least twice the window's possible minimizers, a power of two
    const double est = (double)dw.max_win_bases * 2.0 / (w + 1) * 1.5 + 1024.0;
    int bits = 10;
    while ((double)(1ll << bits) < 2.0 * est && bits < 24) bits++;
    int sms = 0;
    cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_), "attr");
    int grid = std::min(dw.n_windows, sms * 4);
    size_t need = (size_t)grid << bits;
    need *= 8;
    // keep the scratch modest: fewer CTAs for very large windows
    while (need > ((size_t)1 << 31) && grid > sms) {
        grid = std::max(sms, grid / 2);
        need = ((size_t)grid << bits) * 8;
    }
    if (need > tab_bytes_) {
        if (d_tab_) cuda_check(cudaFree(d_tab_), "cudaFree");
        d_tab_ = nullptr;
        cuda_check(cudaMalloc(&d_tab_, need), "cudaMalloc(proposer tables)");
        tab_bytes_ = need;
    }
    bits_out = bits;
    grid_out = grid;
}

void Proposer::plan(const DeviceWindows& dw, int k, int w, std::vector<int32_t>& nodes, std::vector<int64_t>& tb,
                    std::vector<int64_t>& spill, std::vector<float>& cost, std::vector<int64_t>& cells) {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    cudaStream_t s = (cudaStream_t)dw.stream;
    const int64_t nr = std::max<int64_t>(dw.n_reads, 1);
    const size_t fb = 4 * (size_t)nr * T * PROP_CIN, pb = 4 * (size_t)nr * PROP_OUT;
    if (fb > feat_bytes_) {
        if (d_feat_) cuda_check(cudaFree(d_feat_), "cudaFree");
        d_feat_ = nullptr;
        cuda_check(cudaMalloc(&d_feat_, fb), "cudaMalloc(proposer features)");
        feat_bytes_ = fb;
    }
    if (pb > pred_bytes_) {
        if (d_pred_) cuda_check(cudaFree(d_pred_), "cudaFree");
        d_pred_ = nullptr;
        cuda_check(cudaMalloc(&d_pred_, pb), "cudaMalloc(proposer predictions)");
        pred_bytes_ = pb;
    }
    const int nw = dw.n_windows;
    const size_t need = up256(4 * (size_t)nw) + 4 * up256(8 * (size_t)nw);
    if (need > plan_bytes_) {
        if (d_plan_) cuda_check(cudaFree(d_plan_), "cudaFree");
        d_plan_ = nullptr;
        cuda_check(cudaMalloc(&d_plan_, need), "cudaMalloc(proposer plan)");
        plan_bytes_ = need;
    }
    nodes.assign(nw, 0);
    tb.assign(nw, 0);
    spill.assign(nw, 0);
    cost.assign(nw, 0.f);
    cells.assign(nw, 0);
    if (nw == 0) return;
    int bits = 0, grid = 0;
    features_prep(dw, k, w, bits, grid);
    char* p = (char*)d_plan_;
    int32_t* dn = (int32_t*)p;
    int64_t* dt = (int64_t*)(p + up256(4 * (size_t)nw));
    int64_t* ds = (int64_t*)(p + up256(4 * (size_t)nw) + up256(8 * (size_t)nw));
    float* dc = (float*)(p + up256(4 * (size_t)nw) + 2 * up256(8 * (size_t)nw));
    int64_t* dl = (int64_t*)(p + up256(4 * (size_t)nw) + 3 * up256(8 * (size_t)nw));
    // features, inference and plan: recorded once as a CUDA graph per batch shape and
    // replayed with one launch
    const GraphKey key{dw.seq, dw.read_off, dw.read_len, dw.win_off, dw.n_reads, nw, k, w, bits, grid,
                       d_feat_, d_pred_, d_plan_, d_tab_, s};
    if (!graph_exec_ || std::memcmp(&key, &graph_key_, sizeof key) != 0) {
        if (graph_exec_) cudaGraphExecDestroy((cudaGraphExec_t)graph_exec_);
        graph_exec_ = nullptr;
        cudaGraph_t gr = nullptr;
        cuda_check(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "begin capture");
        try {
            features_launch(dw, k, w, bits, grid, d_feat_, s);
            predict_device(d_feat_, dw.n_reads, d_pred_, s);
            k_plan<<<grid_of(nw), 256, 0, s>>>(d_pred_, dw.read_len, dw.win_off, nw, d_extra_, dn, dt, ds, dc, dl);
            cuda_check(cudaGetLastError(), "k_plan");
        } catch (...) {
            cudaStreamEndCapture(s, &gr);
            if (gr) cudaGraphDestroy(gr);
            throw;
        }
        cuda_check(cudaStreamEndCapture(s, &gr), "end capture");
        cudaGraphExec_t ex = nullptr;
        const cudaError_t e = cudaGraphInstantiate(&ex, gr, 0);
        cudaGraphDestroy(gr);
        cuda_check(e, "graph instantiate");
        graph_exec_ = ex;
        std::memcpy(&graph_key_, &key, sizeof key);
    }
    cuda_check(cudaGraphLaunch((cudaGraphExec_t)graph_exec_, s), "graph launch");
    cuda_check(cudaMemcpyAsync(nodes.data(), dn, 4 * (size_t)nw, cudaMemcpyDeviceToHost, s), "D2H plan");
    cuda_check(cudaMemcpyAsync(tb.data(), dt, 8 * (size_t)nw, cudaMemcpyDeviceToHost, s), "D2H plan");
    cuda_check(cudaMemcpyAsync(spill.data(), ds, 8 * (size_t)nw, cudaMemcpyDeviceToHost, s), "D2H plan");
    cuda_check(cudaMemcpyAsync(cost.data(), dc, 4 * (size_t)nw, cudaMemcpyDeviceToHost, s), "D2H plan");
    cuda_check(cudaMemcpyAsync(cells.data(), dl, 8 * (size_t)nw, cudaMemcpyDeviceToHost, s), "D2H plan");
    cuda_check(cudaStreamSynchronize(s), "proposer plan");
}

}  // namespace pb

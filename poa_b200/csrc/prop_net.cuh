// prop_net.cuh - the proposer's network as one kernel: forward pass, and for
// training the whole backward pass, of a tile of reads kept in shared memory.
//
// What bounds it: a read is 32 bins x 64 channels, 1.7 MFLOP forward, so a
// batch is small; run layer by layer (im2col, a GEMM, an elementwise kernel
// per step, ~25 launches a training step) the time was launches, activations
// through memory, and weight-gradient GEMMs whose long sums ran on 1 to 3
// CTAs. Here a CTA holds the weights (BF16) and the activations of 4 reads
// (128 rows), runs every layer there, and keeps its weight gradients in
// registers until its tiles are done; a second kernel adds the CTAs' sums up.
//
// Activations and their gradients are rounded to BF16 between layers, so an
// FP32 sum taken in another order moves some of them to the neighbouring BF16
// value (1 in 10^4; the largest change of a prediction was 9e-4 of its scale
// when the convolutions ran on matrix instructions). The sums that are rounded
// are therefore taken as FP32 multiply-adds in ascending order of the
// contraction, a thread owning one bin of 4 reads x 8 channels; the weight
// gradients, which are not rounded, use m16n8k16 matrix instructions.
//
// A convolution reads rows shifted by its tap, so a read's rows sit between
// two rows of zeros; row strides are odd multiples of 16 bytes, so loads of a
// matrix column are free of bank conflicts.
//
// Measured on a B200, whole calls, layer by layer -> this: the gradient of 256
// reads 4.48 -> 0.17 ms, predictions of 20,000 reads 5.5 -> 2.7 ms (identical;
// ~1 ms of it is the kernel, the rest the copy from pageable host memory). The
// forward multiply-adds bound it: 13 us a tile at an SM's FP32 rate.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "proposer.h"

namespace pb {
namespace net {

typedef __nv_bfloat16 bf16;

constexpr int T = PROP_BINS, CH = PROP_CH, OUT = PROP_OUT;
constexpr int KC1 = PROP_KW * PROP_CIN, KC = PROP_KW * CH;  // convolution widths of layer 1 and of 2, 3
// parameter offsets (floats)
constexpr int OW1 = 0, OB1 = OW1 + CH * KC1;
constexpr int OW2 = OB1 + CH, OB2 = OW2 + CH * KC;
constexpr int OW3 = OB2 + CH, OB3 = OW3 + CH * KC;
constexpr int OW4 = OB3 + CH, OB4 = OW4 + CH * CH;
constexpr int OW5 = OB4 + CH, OB5 = OW5 + OUT * CH;
static_assert(OB5 + OUT == PROP_NPARAM, "parameter layout");
constexpr int X_MEAN = 0, X_STD = 4;

constexpr int RT = 4;                  // reads per tile
constexpr int THREADS = 256;           // 8 warps, 16 rows each
constexpr int PR = T + 2;              // a read's rows with the zero rows around them
constexpr int SY = CH + 8;             // row strides (elements)
constexpr int SX = 40, SWC = KC + 8, SW4 = CH + 8;
constexpr int PART = PROP_NPARAM + 4;  // one CTA's sums: the gradient, then the loss (padded)

struct Smem {
    bf16 xc[RT * T * SX];     // layer 1's input, taps side by side, zero beyond KC1
    bf16 y[3][RT * PR * SY];  // activations; their gradients take their place
    bf16 t1[KC1 * SW4], t2[KC * SW4], t3[KC * SW4];  // convolution weights, [input][output]
    bf16 w2[CH * SWC], w3[CH * SWC];                 // [output][input]
    bf16 w4[CH * SW4], w5[OUT * SW4];
    float b[4 * CH + OUT];
    float h[RT * CH], z[RT * CH], dz[RT * CH];
    float d[RT * OUT];
    float red[THREADS];
};

__device__ __forceinline__ void ldm4t(uint32_t* r, const bf16* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void unpack2(uint32_t u, float& a, float& b) {
    a = __uint_as_float(u << 16);
    b = __uint_as_float(u & 0xffff0000u);
}

// acc[i][j] += sum over k < K, ascending, of a[i * ra + k] * b[k * sb + j]: one bin of
// the tile's reads (ra elements apart) x 8 channels
template <int K>
__device__ __forceinline__ void madd_rows(float (*acc)[8], const bf16* a, int ra, const bf16* b, int sb) {
    for (int k = 0; k < K; k += 4) {
        float x[RT][4];
#pragma unroll
        for (int i = 0; i < RT; i++) {
            const uint2 u = *reinterpret_cast<const uint2*>(a + i * ra + k);
            unpack2(u.x, x[i][0], x[i][1]);
            unpack2(u.y, x[i][2], x[i][3]);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint4 u = *reinterpret_cast<const uint4*>(b + (k + q) * sb);
            float w[8];
            unpack2(u.x, w[0], w[1]);
            unpack2(u.y, w[2], w[3]);
            unpack2(u.z, w[4], w[5]);
            unpack2(u.w, w[6], w[7]);
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(x[i][q], w[j], acc[i][j]);
        }
    }
}

__device__ __forceinline__ uint4 pack8(const float* v) {
    uint4 u;
    __nv_bfloat162 p[4];
#pragma unroll
    for (int j = 0; j < 4; j++) p[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    u.x = *reinterpret_cast<uint32_t*>(&p[0]);
    u.y = *reinterpret_cast<uint32_t*>(&p[1]);
    u.z = *reinterpret_cast<uint32_t*>(&p[2]);
    u.w = *reinterpret_cast<uint32_t*>(&p[3]);
    return u;
}

// relu(acc + bias) as BF16 (at: the thread's bin and channels of the first read)
__device__ __forceinline__ void store_relu(const float (*acc)[8], const float* bias, bf16* at) {
#pragma unroll
    for (int i = 0; i < RT; i++) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = fmaxf(acc[i][j] + bias[j], 0.f);
        *reinterpret_cast<uint4*>(at + i * PR * SY) = pack8(v);
    }
}

// acc masked by y > 0, as BF16, in the place of y
__device__ __forceinline__ void store_masked(const float (*acc)[8], bf16* at) {
#pragma unroll
    for (int i = 0; i < RT; i++) {
        const uint4 u = *reinterpret_cast<const uint4*>(at + i * PR * SY);
        float y[8], v[8];
        unpack2(u.x, y[0], y[1]);
        unpack2(u.y, y[2], y[3]);
        unpack2(u.z, y[4], y[5]);
        unpack2(u.w, y[6], y[7]);
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = y[j] > 0.f ? acc[i][j] : 0.f;
        *reinterpret_cast<uint4*>(at + i * PR * SY) = pack8(v);
    }
}

// Weight gradient of a convolution over the tile: C[o][k*64 + c] += sum over rows of
// dy[row][o] * x[row + k - 1][c]. A warp owns 16 outputs x 96 columns.
__device__ __forceinline__ void conv_wgrad(float (*c)[4], const bf16* dy, const bf16* x, int wid, int lane) {
    const int m0 = (wid & 3) * 16, c0 = (wid >> 2) * 96;
    for (int q = 0; q < 2 * RT; q++) {
        const int row = (q >> 1) * PR + 1 + (q & 1) * 16;
        uint32_t fa[4], fb[4];
        ldm4t(fa, dy + (row + (lane & 7) + ((lane >> 4) & 1) * 8) * SY + m0 + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int n = 0; n < 6; n++) {
            const int col = c0 + n * 16;
            ldm4t(fb, x + (row + col / CH - 1 + (lane & 7) + ((lane >> 3) & 1) * 8) * SY + col % CH + ((lane >> 4) & 1) * 8);
            mma(c[2 * n], fa, fb);
            mma(c[2 * n + 1], fa, fb + 2);
        }
    }
}

__device__ __forceinline__ float read_colsum(const bf16* y, int read, int c) {
    float s = 0.f;
    for (int t = 0; t < T; t++) s += __bfloat162float(y[(read * PR + 1 + t) * SY + c]);
    return s;
}

// Reads idx[0 .. n) (idx == nullptr: 0 .. n) of X [.][T][CIN]. GRAD: loss and
// gradient against the raw targets Y, one CTA's sums to part[blockIdx.x][PART];
// else raw outputs to out [n][OUT].
template <bool GRAD>
__global__ void __launch_bounds__(THREADS, 1) k_net(const float* __restrict__ X, const float* __restrict__ Y,
                                                    const int32_t* __restrict__ idx, int64_t n, const bf16* __restrict__ W,
                                                    const float* __restrict__ Wf, const float* __restrict__ extra,
                                                    float* __restrict__ out, float* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char raw[];
    Smem& s = *reinterpret_cast<Smem*>(raw);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bf16 zero = __float2bfloat16(0.f);
    for (int i = tid; i < CH * KC1; i += THREADS) s.t1[i % KC1 * SW4 + i / KC1] = W[OW1 + i];
    for (int i = tid; i < CH * KC; i += THREADS) {
        const int o = i / KC, k = i % KC;
        const bf16 a = W[OW2 + i], b = W[OW3 + i];
        s.t2[k * SW4 + o] = a;
        s.t3[k * SW4 + o] = b;
        if (GRAD) {
            s.w2[o * SWC + k] = a;
            s.w3[o * SWC + k] = b;
        }
    }
    for (int i = tid; i < CH * CH; i += THREADS) s.w4[i / CH * SW4 + i % CH] = W[OW4 + i];
    for (int i = tid; i < OUT * CH; i += THREADS) s.w5[i / CH * SW4 + i % CH] = W[OW5 + i];
    for (int i = tid; i < 4 * CH + OUT; i += THREADS) {
        const int off[5] = {OB1, OB2, OB3, OB4, OB5};
        s.b[i] = Wf[off[i / CH] + i % CH];
    }
    for (int i = tid; i < 3 * RT * 2 * SY; i += THREADS) {  // the zero rows
        const int a = i / (RT * 2 * SY), q = i / SY % (RT * 2);
        s.y[a][((q >> 1) * PR + (q & 1) * (PR - 1)) * SY + i % SY] = zero;
    }
    float g3[12][4], g2[12][4], g1[2][4], g4[16], g5 = 0.f, gb[4] = {0.f, 0.f, 0.f, 0.f}, gb5 = 0.f, loss = 0.f;
    if (GRAD) {
#pragma unroll
        for (int i = 0; i < 12; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) g3[i][j] = g2[i][j] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) g1[0][j] = g1[1][j] = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) g4[i] = 0.f;
    }
    const int bin = tid >> 3, n0 = (tid & 7) * 8;     // the convolutions: one bin of every read x 8 channels
    const int at = (1 + bin) * SY + n0;               // ... in the padded arrays, first read
    const int qr = tid >> 6, qc = tid & 63;           // (read, channel) of the per-read steps
    for (int64_t tile = blockIdx.x; tile * RT < n; tile += gridDim.x) {
        __syncthreads();
        const int have = (int)(n - tile * RT < RT ? n - tile * RT : RT);
        for (int i = tid; i < RT * T * SX; i += THREADS) {
            const int r = i / SX, k = i % SX, q = r / T, tt = r % T + k / PROP_CIN - 1;
            float v = 0.f;
            if (k < KC1 && q < have && tt >= 0 && tt < T) {
                const int64_t src = idx ? idx[tile * RT + q] : tile * RT + q;
                v = X[(src * T + tt) * PROP_CIN + k % PROP_CIN];
            }
            s.xc[i] = __float2bfloat16(v);
        }
        __syncthreads();
        float c[RT][8];
        auto clear = [&] {
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) c[i][j] = 0.f;
        };
        clear();
        madd_rows<KC1>(c, s.xc + bin * SX, T * SX, s.t1 + n0, SW4);
        store_relu(c, s.b + n0, s.y[0] + at);
        __syncthreads();
        for (int layer = 1; layer < 3; layer++) {
            clear();
            const bf16* t = (layer == 1 ? s.t2 : s.t3) + n0;
            for (int k = 0; k < PROP_KW; k++)
                madd_rows<CH>(c, s.y[layer - 1] + (bin + k) * SY, PR * SY, t + k * CH * SW4, SW4);
            store_relu(c, s.b + layer * CH + n0, s.y[layer] + at);
            __syncthreads();
        }
        // mean over the bins, the dense layers (per read, plain FP32)
        s.h[tid] = __bfloat162float(__float2bfloat16(read_colsum(s.y[2], qr, qc) * (1.f / T)));
        __syncthreads();
        {
            float v = 0.f;
            for (int k = 0; k < CH; k++) v = fmaf(s.h[qr * CH + k], __bfloat162float(s.w4[qc * SW4 + k]), v);
            s.z[tid] = __bfloat162float(__float2bfloat16(fmaxf(v + s.b[3 * CH + qc], 0.f)));
        }
        __syncthreads();
        if (tid < RT * OUT) {
            const int q = tid / OUT, o = tid % OUT;
            float v = 0.f;
            for (int k = 0; k < CH; k++) v = fmaf(s.z[q * CH + k], __bfloat162float(s.w5[o * SW4 + k]), v);
            v += s.b[4 * CH + o];
            const int64_t rn = tile * RT + q;
            if (!GRAD) {
                if (q < have) out[rn * OUT + o] = v * extra[X_STD + o] + extra[X_MEAN + o];
            } else {
                float d = 0.f;
                const float scale = 1.f / (float)(n * OUT);
                if (q < have) d = v - (Y[(idx ? (int64_t)idx[rn] : rn) * OUT + o] - extra[X_MEAN + o]) / extra[X_STD + o];
                loss += d * d * scale;
                s.d[tid] = __bfloat162float(__float2bfloat16(2.f * d * scale));
            }
        }
        if (!GRAD) continue;
        __syncthreads();
        // dense layers
        {
            float dz = 0.f;
#pragma unroll
            for (int q = 0; q < RT; q++) g5 = fmaf(s.d[q * OUT + qr], s.z[q * CH + qc], g5);  // (output qr, channel qc)
#pragma unroll
            for (int o = 0; o < OUT; o++) dz = fmaf(s.d[qr * OUT + o], __bfloat162float(s.w5[o * SW4 + qc]), dz);
            s.dz[tid] = __bfloat162float(__float2bfloat16(s.z[tid] > 0.f ? dz : 0.f));
            if (tid < OUT)
                for (int q = 0; q < RT; q++) gb5 += s.d[q * OUT + tid];
        }
        __syncthreads();
        {
            float dh = 0.f;
            for (int o = 0; o < CH; o++) dh = fmaf(s.dz[qr * CH + o], __bfloat162float(s.w4[o * SW4 + qc]), dh);
#pragma unroll
            for (int i = 0; i < 16; i++)
#pragma unroll
                for (int q = 0; q < RT; q++) g4[i] = fmaf(s.dz[q * CH + qr * 16 + i], s.h[q * CH + qc], g4[i]);
            gb[3] += s.dz[tid];
            const bf16 v = __float2bfloat16(dh * (1.f / T));
            float sum = 0.f;
            for (int t = 0; t < T; t++) {
                bf16* y = s.y[2] + (qr * PR + 1 + t) * SY + qc;
                const bf16 dv = __bfloat162float(*y) > 0.f ? v : zero;
                *y = dv;
                sum += __bfloat162float(dv);
            }
            gb[2] += sum;
        }
        __syncthreads();
        // convolutions 3 and 2: weight gradient, then the gradient of the layer below in its place
#pragma unroll
        for (int layer = 2; layer > 0; layer--) {
            conv_wgrad(layer == 2 ? g3 : g2, s.y[layer], s.y[layer - 1], wid, lane);
            float sum[RT][8];
            for (int k = 0; k < PROP_KW; k++) {
                clear();
                madd_rows<CH>(c, s.y[layer] + (bin + 2 - k) * SY, PR * SY, (layer == 2 ? s.w3 : s.w2) + k * CH + n0, SWC);
#pragma unroll
                for (int i = 0; i < RT; i++)
#pragma unroll
                    for (int j = 0; j < 8; j++) sum[i][j] = k == 0 ? c[i][j] : sum[i][j] + c[i][j];
            }
            __syncthreads();
            store_masked(sum, s.y[layer - 1] + at);
            __syncthreads();
            gb[layer - 1] += read_colsum(s.y[layer - 1], qr, qc);
        }
        {
            const int m0 = (wid & 3) * 16, c0 = (wid >> 2) * 16;
            for (int q = 0; q < 2 * RT; q++) {
                const int r = (q >> 1) * PR + 1 + (q & 1) * 16;
                uint32_t fa[4], fb[4];
                ldm4t(fa, s.y[0] + (r + (lane & 7) + ((lane >> 4) & 1) * 8) * SY + m0 + ((lane >> 3) & 1) * 8);
                ldm4t(fb, s.xc + (q * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * SX + c0 + ((lane >> 4) & 1) * 8);
                mma(g1[0], fa, fb);
                mma(g1[1], fa, fb + 2);
            }
        }
    }
    if (!GRAD) return;
    float* p = part + (int64_t)blockIdx.x * PART;
    const int m0 = (wid & 3) * 16 + (lane >> 2), l0 = (lane & 3) * 2;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int o = m0 + (j >> 1) * 8, cc = l0 + (j & 1);
#pragma unroll
        for (int i = 0; i < 12; i++) {
            p[OW3 + o * KC + (wid >> 2) * 96 + i * 8 + cc] = g3[i][j];
            p[OW2 + o * KC + (wid >> 2) * 96 + i * 8 + cc] = g2[i][j];
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int col = (wid >> 2) * 16 + i * 8 + cc;
            if (col < KC1) p[OW1 + o * KC1 + col] = g1[i][j];
        }
    }
#pragma unroll
    for (int i = 0; i < 16; i++) p[OW4 + (qr * 16 + i) * CH + qc] = g4[i];
    p[OW5 + tid] = g5;
    const int ob[4] = {OB1, OB2, OB3, OB4};
#pragma unroll
    for (int b = 0; b < 4; b++) {  // per (read slot, channel): the four slots together
        __syncthreads();
        s.red[tid] = gb[b];
        __syncthreads();
        if (tid < CH) p[ob[b] + tid] = s.red[tid] + s.red[CH + tid] + s.red[2 * CH + tid] + s.red[3 * CH + tid];
    }
    if (tid < OUT) p[OB5 + tid] = gb5;
    __syncthreads();
    s.red[tid] = tid < RT * OUT ? loss : 0.f;
    __syncthreads();
    if (tid == 0) {
        float l = 0.f;
        for (int i = 0; i < RT * OUT; i++) l += s.red[i];
        p[PROP_NPARAM] = l;
    }
}

// g[i] = sum over the CTAs' parts; *loss += their losses
__global__ void k_net_sum(const float* __restrict__ part, int ctas, float* __restrict__ g, float* __restrict__ loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > PROP_NPARAM) return;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < ctas; c += 8)
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (c + q < ctas) s[q] += part[(int64_t)(c + q) * PART + i];
    const float v = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
    if (i < PROP_NPARAM) g[i] = v;
    else *loss += v;
}

}  // namespace net
}  // namespace pb

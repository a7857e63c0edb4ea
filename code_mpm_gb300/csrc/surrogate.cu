// Learned von Mises hardening return map: training samples from the exact
// FP64 map, FP32 training kernels (forward, backward, Adam), and the BF16
// tcgen05 inference kernel.  The network replaces
// ConstitutiveRelation::calculateIncrement_VonMisesHardening
// (ConstitutiveRelation_calculateIncrement_VonMisesHardening.cpp:4-92) for
// clearly plastic trial states; it is this library's addition.
//
// Network: x (13 inputs, padded to 16) -> 128 -> 128 -> 128 (ReLU) -> 8 (7
// used).  ReLU rather than a smooth activation: its inference epilogue is a
// bias add and one packed convert per two values, with nothing on the
// special-function pipe, so the epilogue keeps pace with the tensor core.
// Inputs are scaled to O(1): stress and R by 1/yield, the strain
// increment by 1/deps_sigma; outputs are standardised by the training set's
// mean and standard deviation.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "mpm_surrogate.h"
#include "physics.cuh"
#include "surrogate.cuh"

namespace mpm {
namespace net {

constexpr int IN = 16, NIN = 13, HID = 128, OUT = 8, NOUT = 7;
constexpr long long OW1 = 0, OB1 = OW1 + HID * IN, OW2 = OB1 + HID, OB2 = OW2 + HID * HID, OW3 = OB2 + HID,
                    OB3 = OW3 + HID * HID, OW4 = OB3 + HID, OB4 = OW4 + OUT * HID, NPARAM = OB4 + OUT;

#define NCK(x)                                      \
    do {                                            \
        cudaError_t e_ = (x);                       \
        if (e_ != cudaSuccess) {                    \
            cudaGetLastError();                     \
            return MPM_ERR_CUDA;                    \
        }                                           \
    } while (0)

// ---------------------------------------------------------------------------
// counter-based random numbers (splitmix64 finaliser of (seed, sample, draw))
// ---------------------------------------------------------------------------
__host__ __device__ inline uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}
__device__ inline float uni(uint64_t seed, uint64_t i, uint32_t j) {
    uint64_t h = mix64(seed + 0x9e3779b97f4a7c15ULL * (i * 64 + j + 1));
    return ((float)(h >> 40) + 0.5f) * (1.0f / 16777216.0f);  // (0, 1)
}
__device__ inline float gauss(uint64_t seed, uint64_t i, uint32_t j) {
    float u1 = uni(seed, i, 2 * j + 32), u2 = uni(seed, i, 2 * j + 33);
    return sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
}

struct SampleCfg {
    double yield, range, epmax, dsig, C0, C1;
    uint64_t seed;
    int sampling;
};

// One sample: prior stress U(+-range yield), R from the closed form of the
// hardening law for a uniform equivalent plastic strain
// (R = sqrt(2/3) C1 (1 - exp(-C0 epbar)), the solution of dR = C0 (sqrt(2/3)
// C1 - R) depbar), strain increment N(0, dsig); target = the exact FP64
// return map (cr_increment<double>).  x: normalised inputs (16, zero padded),
// raw: physical inputs (13), t: physical outputs (7) and f_trial / k0.
__device__ void label_sample(long long i, const double sig[6], double R, const double e[6], const SampleCfg& sc,
                             const MatConst& M, float* __restrict__ x, float* __restrict__ t);

__global__ void k_generate(long long n, long long i0, SampleCfg sc, MatConst M, float* __restrict__ x,
                           float* __restrict__ t) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t gi = (uint64_t)(i0 + i);
    double sig[6], e[6];
    const double ep = uni(sc.seed, gi, 6) * sc.epmax;
    const double R = sqrt(2.0 / 3.0) * sc.C1 * (1.0 - exp(-sc.C0 * ep));
    if (sc.sampling == 0) {
        for (int c = 0; c < 6; ++c) sig[c] = (2.0 * uni(sc.seed, gi, c) - 1.0) * sc.range * sc.yield;
    } else {
        // a random deviator scaled to sqrt J2 = U(0.85, 1) (k0 + R/sqrt 2), plus a hydrostatic part
        double d[6];
        for (int c = 0; c < 6; ++c) d[c] = gauss(sc.seed, gi, 8 + c);
        const double h = (d[0] + d[1] + d[2]) / 3.0;
        for (int c = 0; c < 3; ++c) d[c] -= h;
        const double j2 = ((d[0] - d[1]) * (d[0] - d[1]) + (d[1] - d[2]) * (d[1] - d[2]) + (d[2] - d[0]) * (d[2] - d[0])) /
                              6.0 + d[3] * d[3] + d[4] * d[4] + d[5] * d[5];
        const double rad = M.k0 + R * 0.70710678118654752440;
        const double sc2 = (0.85 + 0.15 * uni(sc.seed, gi, 7)) * rad / sqrt(j2);
        const double p = (2.0 * uni(sc.seed, gi, 5) - 1.0) * sc.yield;
        for (int c = 0; c < 6; ++c) sig[c] = d[c] * sc2 + (c < 3 ? p : 0.0);
    }
    for (int c = 0; c < 6; ++c) e[c] = gauss(sc.seed, gi, c) * sc.dsig;
    label_sample(i, sig, R, e, sc, M, x, t);
}

// Samples given as physical input rows (e.g. harvested from a run of the
// plain method): labelled by the exact FP64 map like generated ones.
__global__ void k_label_rows(long long n, const float* __restrict__ in, SampleCfg sc, MatConst M,
                             float* __restrict__ x, float* __restrict__ t) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double sig[6], e[6];
    for (int c = 0; c < 6; ++c) {
        sig[c] = in[i * NIN + c];
        e[c] = in[i * NIN + 7 + c];
    }
    label_sample(i, sig, (double)in[i * NIN + 6], e, sc, M, x, t);
}

// normalised inputs x[i] (16) and targets t[i] (plastic correction, dR, f_trial / k0)
__device__ void label_sample(long long i, const double sig[6], double R, const double e[6], const SampleCfg& sc,
                             const MatConst& M, float* __restrict__ x, float* __restrict__ t) {
    CrOut<double> o;
    cr_increment<double>(M, R, sig, e, o);
    // trial yield function (…_VonMisesHardening.cpp:35-46)
    double dtr[6];
    trial_increment<double>(M, e, dtr);
    double tr[6];
    for (int c = 0; c < 6; ++c) tr[c] = sig[c] + dtr[c];
    const double a01 = tr[0] - tr[1], a12 = tr[1] - tr[2], a20 = tr[2] - tr[0];
    const double J2 = (a01 * a01 + a12 * a12 + a20 * a20) / 6.0 + tr[3] * tr[3] + tr[4] * tr[4] + tr[5] * tr[5];
    const double f = sqrt(J2) - (M.k0 + R * 0.70710678118654752440);
    float* xi = x + i * IN;
    for (int c = 0; c < 6; ++c) {
        xi[c] = (float)(sig[c] / sc.yield);
        xi[7 + c] = (float)(e[c] / sc.dsig);
    }
    xi[6] = (float)(R / sc.yield);
    xi[13] = xi[14] = xi[15] = 0.0f;
    // targets: the plastic correction dsigma - D de (the kernels add D de back)
    float* ti = t + i * OUT;
    for (int c = 0; c < 6; ++c) ti[c] = (float)(o.dsig[c] - dtr[c]);
    ti[6] = (float)o.dR;
    ti[7] = (float)(f / M.k0);
}

// Per-column min and max of the normalised inputs x (n x 16, first NIN
// columns) as order-preserving unsigned keys: box[c] min, box[NIN + c] max.
__device__ __forceinline__ unsigned f2ord(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void k_box(long long n, const float* __restrict__ x, unsigned* __restrict__ box) {
    unsigned lo[NIN], hi[NIN];
    for (int c = 0; c < NIN; ++c) {
        lo[c] = 0xffffffffu;
        hi[c] = 0u;
    }
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        for (int c = 0; c < NIN; ++c) {
            const unsigned k = f2ord(x[i * IN + c]);
            lo[c] = min(lo[c], k);
            hi[c] = max(hi[c], k);
        }
    for (int c = 0; c < NIN; ++c) {
        const unsigned a = __reduce_min_sync(0xffffffffu, lo[c]), b = __reduce_max_sync(0xffffffffu, hi[c]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&box[c], a);
            atomicMax(&box[NIN + c], b);
        }
    }
}

static float ord2f(unsigned k) {
    const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    memcpy(&f, &u, 4);
    return f;
}

// per-output sums of the targets (mean and standard deviation)
__global__ void k_moments(long long n, const float* __restrict__ t, double* __restrict__ acc) {
    __shared__ double s[2 * NOUT];
    if (threadIdx.x < 2 * NOUT) s[threadIdx.x] = 0.0;
    __syncthreads();
    double a[NOUT] = {}, b[NOUT] = {};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        for (int c = 0; c < NOUT; ++c) {
            double v = t[i * OUT + c];
            a[c] += v;
            b[c] += v * v;
        }
    for (int c = 0; c < NOUT; ++c) {
        atomicAdd(&s[c], a[c]);
        atomicAdd(&s[NOUT + c], b[c]);
    }
    __syncthreads();
    if (threadIdx.x < 2 * NOUT) atomicAdd(&acc[threadIdx.x], s[threadIdx.x]);
}

__global__ void k_normalise_targets(long long n, const float* __restrict__ t, const float* __restrict__ shift,
                                    const float* __restrict__ inv_scale, float* __restrict__ tn) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int c = 0; c < NOUT; ++c) tn[i * OUT + c] = (t[i * OUT + c] - shift[c]) * inv_scale[c];
    tn[i * OUT + 7] = 0.0f;
}

// ---------------------------------------------------------------------------
// FP32 training kernels.  A batch of n rows goes through
//   forward   h = relu(x W^T + b), three layers          k_layer<true>
//   head      y = h3 W4^T + b4, the loss, dL/dy, and back through layer 4:
//             d3 = (dy W4) relu'(h3), the gradients of W4, b4 and b3   k_head
//   backward  d = (d W) relu'(h), two layers, and the bias gradient of each
//             (the column sums of d, from the tile in registers)  k_layer<false>
//   weights   dW += d^T h, split over the rows                      k_weight_grad
// relu'(z) is taken from h (z > 0 exactly where h = relu(z) > 0), so the
// pre-activations are not stored.
//
// The GEMMs are bound by the FP32 FMAs: a block of 256 threads forms a 128 x
// 128 tile, 8 x 8 outputs per thread in four 4 x 4 quarters (each thread's 16
// operand values per k are four 16-byte shared loads for 64 FMAs), the next
// 16-deep slice on its way to registers while the current one is used.  Before,
// with 64 x 64 tiles, 4 x 4 outputs, no overlap, stored pre-activations and
// separate kernels for layer 4, the loss and the column sums, a batch of 65,536
// took 928 us through mpm_net_loss_grad, 1,000 rows 340 us; now 428 and 140.
// ---------------------------------------------------------------------------
constexpr int GT = 256;       // threads
constexpr int GK = 16;        // slice depth
constexpr int GS = HID + 4;   // shared row stride

struct GemmTile {
    float a[2][GK][GS], b[2][GK][GS];
};

// acc[i][j]: rows ty * 4 + (i & 3) + 64 (i >> 2), columns tx * 4 + (j & 3) + 64 (j >> 2).  Two columns per
// instruction (fma.rn.f32x2, the same roundings as two fmaf): half the issue slots beside the shared loads.
__device__ __forceinline__ void tile_fma(const GemmTile& s, int buf, int ty, int tx, float acc[8][8]) {
    unsigned long long (*acc2)[4] = reinterpret_cast<unsigned long long (*)[4]>(acc);
#pragma unroll
    for (int k = 0; k < GK; ++k) {
        float a[8];
        unsigned long long b[4];
        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&s.a[buf][k][4 * ty]);
        *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&s.a[buf][k][64 + 4 * ty]);
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&s.b[buf][k][4 * tx]);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&s.b[buf][k][64 + 4 * tx]);
        b[0] = b0.x, b[1] = b0.y, b[2] = b1.x, b[3] = b1.y;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            unsigned long long aa;
            asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[i]));
#pragma unroll
            for (int j = 0; j < 4; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2[i][j]) : "l"(aa), "l"(b[j]));
        }
    }
}

// FWD: C = relu(A W^T + bias), A n x K, W 128 x K.
// else: C = (A W) where H > 0 (else 0), A n x 128, W 128 x 128; the column sums of C added to gbias.
template <bool FWD, int K>
__global__ void __launch_bounds__(GT, 2) k_layer(int n, const float* A, const float* __restrict__ W,
                                                 const float* __restrict__ bias, const float* H,
                                                 float* __restrict__ C, float* __restrict__ gbias) {
    extern __shared__ __align__(16) unsigned char net_smem[];
    GemmTile& s = *reinterpret_cast<GemmTile*>(net_smem);
    step_enter<true>();
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int m0 = blockIdx.x * 128;
    // a slice: rows r and r + 64, four k each (stored transposed); W the same, or (backward) k rows of 128
    const int lr = tid >> 2, lk = (tid & 3) * 4, br = tid >> 5, bc = (tid & 31) * 4;
    float4 ra[2], rb[2];
    auto load = [&](int k0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = lr + 64 * h;
            ra[h] = m0 + r < n ? *reinterpret_cast<const float4*>(A + (long long)(m0 + r) * K + k0 + lk)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
            rb[h] = FWD ? *reinterpret_cast<const float4*>(W + r * K + k0 + lk)
                        : *reinterpret_cast<const float4*>(W + (k0 + br + 8 * h) * HID + bc);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = lr + 64 * h;
            const float va[4] = {ra[h].x, ra[h].y, ra[h].z, ra[h].w}, vb[4] = {rb[h].x, rb[h].y, rb[h].z, rb[h].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) s.a[buf][lk + j][r] = va[j];
            if (FWD) {
#pragma unroll
                for (int j = 0; j < 4; ++j) s.b[buf][lk + j][r] = vb[j];
            } else {
                *reinterpret_cast<float4*>(&s.b[buf][br + 8 * h][bc]) = rb[h];
            }
        }
    };
    __align__(8) float acc[8][8] = {};
    load(0);
    store(0);
    if (GK < K) load(GK);  // each slice is requested before the barrier in front of the one it follows
    __syncthreads();
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += GK) {
        const int buf = (k0 / GK) & 1;
        tile_fma(s, buf, ty, tx, acc);
        if (k0 + GK < K) store(buf ^ 1);
        if (k0 + 2 * GK < K) load(k0 + 2 * GK);
        __syncthreads();
    }
    float cs[8] = {};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + 4 * ty + (i & 3) + 64 * (i >> 2);
        if (m >= n) continue;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int c = 4 * tx + 64 * q;
            const long long o = (long long)m * HID + c;
            float v[4];
            if (FWD) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = fmaxf(acc[i][4 * q + j] + bias[c + j], 0.0f);
            } else {
                const float4 h = *reinterpret_cast<const float4*>(H + o);
                const float hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = hv[j] > 0.0f ? acc[i][4 * q + j] : 0.0f;
                    cs[4 * q + j] += v[j];
                }
            }
            *reinterpret_cast<float4*>(C + o) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
    if (!FWD) {  // the tile's column sums: over ty in shared memory, then one atomic per column
#pragma unroll
        for (int j = 0; j < 8; ++j) s.a[0][ty][4 * tx + (j & 3) + 64 * (j >> 2)] = cs[j];
        __syncthreads();
        if (tid < HID) {
            float v = 0.0f;
#pragma unroll
            for (int r = 0; r < 16; ++r) v += s.a[0][r][tid];
            atomicAdd(&gbias[tid], v);
        }
    }
}

// gW[128 x N] += D^T X over this block's rows (D n x 128, X n x N), N = 128 or 16.
template <int N>
__global__ void __launch_bounds__(GT, 2) k_weight_grad(int n, int rows, const float* D,
                                                       const float* X, float* __restrict__ gW) {
    static_assert(N == HID || N == IN, "layer widths");
    extern __shared__ __align__(16) unsigned char net_smem[];
    GemmTile& s = *reinterpret_cast<GemmTile*>(net_smem);
    step_enter<true>();
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, br = tid >> 5, bc = (tid & 31) * 4;
    const int beg = blockIdx.x * rows, end = min(n, beg + rows);
    float4 rd[2], rx[2];
    auto load = [&](int r0) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = r0 + br + 8 * h;
            rd[h] = r < end ? *reinterpret_cast<const float4*>(D + (long long)r * HID + bc) : z;
            if (N == HID) rx[h] = r < end ? *reinterpret_cast<const float4*>(X + (long long)r * HID + bc) : z;
        }
        if (N == IN) {  // 16 rows of 16: the first 64 threads
            const int r = r0 + (tid >> 2);
            rx[0] = tid < 64 && r < end ? *reinterpret_cast<const float4*>(X + (long long)r * IN + (tid & 3) * 4) : z;
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            *reinterpret_cast<float4*>(&s.a[buf][br + 8 * h][bc]) = rd[h];
            if (N == HID) *reinterpret_cast<float4*>(&s.b[buf][br + 8 * h][bc]) = rx[h];
        }
        if (N == IN && tid < 64) *reinterpret_cast<float4*>(&s.b[buf][tid >> 2][(tid & 3) * 4]) = rx[0];
    };
    __align__(8) float acc[8][8] = {};  // N = 16: acc[i][0] of column tx
    load(beg);
    store(0);
    if (beg + GK < end) load(beg + GK);
    __syncthreads();
    int buf = 0;
#pragma unroll 1
    for (int r0 = beg; r0 < end; r0 += GK, buf ^= 1) {
        if constexpr (N == HID) {
            tile_fma(s, buf, ty, tx, acc);
        } else {
#pragma unroll
            for (int k = 0; k < GK; ++k) {
                const float b = s.b[buf][k][tx];
                const float4 a0 = *reinterpret_cast<const float4*>(&s.a[buf][k][4 * ty]);
                const float4 a1 = *reinterpret_cast<const float4*>(&s.a[buf][k][64 + 4 * ty]);
                const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][0] = fmaf(a[i], b, acc[i][0]);
            }
        }
        if (r0 + GK < end) store(buf ^ 1);
        if (r0 + 2 * GK < end) load(r0 + 2 * GK);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float* g = gW + (4 * ty + (i & 3) + 64 * (i >> 2)) * N;
        if constexpr (N == HID) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
                atomicAdd(reinterpret_cast<float4*>(g + 4 * tx + 64 * q),
                          make_float4(acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2], acc[i][4 * q + 3]));
        } else {
            atomicAdd(g + tx, acc[i][0]);
        }
    }
}

// The output layer, a warp per row (lane l holds columns 4l .. 4l + 3).
// GRAD: also the loss (mean over the batch and the 7 used outputs), dL/dy and
// layer 4's backward pass: d = (dy W4) where h > 0, gradients of W4, b4 and,
// as the column sums of d, of layer 3's bias; without it y is written.
constexpr int HEAD_WARPS = 16;
template <bool GRAD>
__global__ void __launch_bounds__(HEAD_WARPS * 32) k_head(long long n, const float* h,
                                                          const float* __restrict__ W4, const float* __restrict__ b4,
                                                          const float* t, float* __restrict__ y,
                                                          float* __restrict__ d, float* __restrict__ gW4,
                                                          float* __restrict__ gb4, float* __restrict__ gb3,
                                                          double* __restrict__ loss) {
    __shared__ float sg[OUT * HID + HID + OUT];
    step_enter<true>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (GRAD) {
        for (int i = threadIdx.x; i < OUT * HID + HID + OUT; i += blockDim.x) sg[i] = 0.0f;
        __syncthreads();
    }
    float w[OUT][4], gw[OUT][4] = {}, gs[4] = {}, gb = 0.0f;
#pragma unroll
    for (int c = 0; c < OUT; ++c) *reinterpret_cast<float4*>(w[c]) = *reinterpret_cast<const float4*>(W4 + c * HID + 4 * lane);
    // after the halving exchange below a lane holds output c
    const int c = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    const float bc = b4[c], sc = 2.0f / (float)(n * NOUT);
    double l = 0.0;
    // two rows' loads ahead of the row in hand
    const long long step = (long long)gridDim.x * HEAD_WARPS, r0 = blockIdx.x * (long long)HEAD_WARPS + warp;
    float4 hn[2];
    float tn[2];
    auto fetch = [&](int q, long long r) {
        hn[q] = r < n ? *reinterpret_cast<const float4*>(h + r * HID + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        tn[q] = GRAD && r < n ? t[r * OUT + c] : 0.0f;
    };
    fetch(0, r0);
    fetch(1, r0 + step);
    for (long long r = r0; r < n; r += step) {
        const float hv[4] = {hn[0].x, hn[0].y, hn[0].z, hn[0].w}, tv = tn[0];
        hn[0] = hn[1];
        tn[0] = tn[1];
        fetch(1, r + 2 * step);
        float p[OUT];
#pragma unroll
        for (int k = 0; k < OUT; ++k) p[k] = w[k][0] * hv[0] + w[k][1] * hv[1] + w[k][2] * hv[2] + w[k][3] * hv[3];
        // eight sums over the warp: halve the outputs a lane keeps with each exchange
#pragma unroll
        for (int half = 4, off = 16; half; half >>= 1, off >>= 1) {
            const bool up = lane & off;
#pragma unroll
            for (int k = 0; k < half; ++k) {
                const float send = up ? p[k] : p[half + k], keep = up ? p[half + k] : p[k];
                p[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
            }
        }
        float v = p[0];
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += bc;
        if (!GRAD) {
            if ((lane & 3) == 0) y[r * OUT + c] = v;
            continue;
        }
        const float diff = c < NOUT ? v - tv : 0.0f, dy = sc * diff;
        l += (double)diff * diff;
        gb += dy;
        float o[4] = {};
#pragma unroll
        for (int k = 0; k < OUT; ++k) {
            const float g = __shfl_sync(0xffffffffu, dy, ((k & 4) ? 16 : 0) | ((k & 2) ? 8 : 0) | ((k & 1) ? 4 : 0));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[j] = fmaf(g, w[k][j], o[j]);
                gw[k][j] = fmaf(g, hv[j], gw[k][j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            o[j] = hv[j] > 0.0f ? o[j] : 0.0f;
            gs[j] += o[j];
        }
        *reinterpret_cast<float4*>(d + r * HID + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
    }
    if (!GRAD) return;
    // the block's sums, then one atomic per parameter
#pragma unroll
    for (int k = 0; k < OUT; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) atomicAdd(&sg[k * HID + 4 * lane + j], gw[k][j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) atomicAdd(&sg[OUT * HID + 4 * lane + j], gs[j]);
    if ((lane & 3) == 0) atomicAdd(&sg[OUT * HID + HID + c], gb);
    l = (lane & 3) == 0 ? l : 0.0;
    for (int o = 16; o; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    if (lane == 0) atomicAdd(loss, l / (double)(n * NOUT));
    __syncthreads();
    for (int i = threadIdx.x; i < OUT * HID; i += blockDim.x) atomicAdd(&gW4[i], sg[i]);
    if (threadIdx.x < HID) atomicAdd(&gb3[threadIdx.x], sg[OUT * HID + threadIdx.x]);
    if (threadIdx.x < OUT) atomicAdd(&gb4[threadIdx.x], sg[OUT * HID + HID + threadIdx.x]);
}

// A training kernel (they begin with step_enter): its launch overlaps the kernel before it.
template <typename... Ex, typename... Act>
static void launch_net(cudaStream_t s, void (*kernel)(Ex...), long long grid, unsigned block, size_t smem, Act&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}

__global__ void k_adam(long long n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// rows of the training set in a pseudo-random order: row j of the epoch is
// (a j + c) mod n with a coprime to n (a full-period affine permutation)
__global__ void k_gather(long long n, const float* __restrict__ x, const float* __restrict__ t, long long a,
                         long long c, long long j0, int rows, float* __restrict__ xb, float* __restrict__ tb) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const unsigned long long j = (unsigned long long)(j0 + r);
    const long long i = (long long)(((unsigned __int128)a * j + (unsigned long long)c) % (unsigned long long)n);
    const float4* xs = reinterpret_cast<const float4*>(x + i * IN);
    float4* xd = reinterpret_cast<float4*>(xb + (long long)r * IN);
#pragma unroll
    for (int k = 0; k < 4; ++k) xd[k] = xs[k];
    const float4* ts = reinterpret_cast<const float4*>(t + i * OUT);
    float4* td = reinterpret_cast<float4*>(tb + (long long)r * OUT);
    td[0] = ts[0];
    td[1] = ts[1];
}

// validation errors in physical units: sums of squared dstress/yield errors
// (all samples, and those outside the fallback band), max outside the band,
// squared dR/yield errors
__global__ void k_val_errors(long long n, const float* __restrict__ yn, const float* __restrict__ t,
                             const float* __restrict__ shift, const float* __restrict__ scale, float inv_yield,
                             float band, double* __restrict__ acc, unsigned* __restrict__ maxbits) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    double s_all = 0, s_out = 0, s_r = 0, cnt_out = 0;
    float mx = 0.0f;
    if (i < n) {
        const bool outside = fabsf(t[i * OUT + 7]) >= band;
        for (int c = 0; c < 6; ++c) {
            const float y = yn[i * OUT + c] * scale[c] + shift[c];
            const float d = (y - t[i * OUT + c]) * inv_yield;
            s_all += (double)d * d;
            if (outside) {
                s_out += (double)d * d;
                mx = fmaxf(mx, fabsf(d));
            }
        }
        const float yr = yn[i * OUT + 6] * scale[6] + shift[6];
        const float dr = (yr - t[i * OUT + 6]) * inv_yield;
        s_r = (double)dr * dr;
        cnt_out = outside ? 1.0 : 0.0;
    }
    for (int o = 16; o; o >>= 1) {
        s_all += __shfl_down_sync(0xffffffffu, s_all, o);
        s_out += __shfl_down_sync(0xffffffffu, s_out, o);
        s_r += __shfl_down_sync(0xffffffffu, s_r, o);
        cnt_out += __shfl_down_sync(0xffffffffu, cnt_out, o);
        mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&acc[0], s_all);
        atomicAdd(&acc[1], s_out);
        atomicAdd(&acc[2], s_r);
        atomicAdd(&acc[3], cnt_out);
        atomicMax(maxbits, __float_as_uint(mx));
    }
}

// physical inputs (n x 13) -> normalised rows (n x 16)
__global__ void k_norm_inputs(long long n, const float* __restrict__ in, const float* __restrict__ inv_scale,
                              float* __restrict__ x) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int c = 0; c < NIN; ++c) x[i * IN + c] = in[i * NIN + c] * inv_scale[c];
    x[i * IN + 13] = x[i * IN + 14] = x[i * IN + 15] = 0.0f;
}

// the elastic predictor D de of physical input row `in` (trial_increment, FP32)
__device__ __forceinline__ void elastic_predictor(const MatConst& M, const float* in, float d[6]) {
    float e[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) e[c] = in[7 + c];
    trial_increment<float>(M, e, d);
}

// normalised outputs (n x 8) -> physical (n x 7): correction + D de, dR
__global__ void k_denorm_outputs(long long n, const float* __restrict__ yn, const float* __restrict__ scale,
                                 const float* __restrict__ shift, const float* __restrict__ in, MatConst M,
                                 float* __restrict__ out) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float d[6];
    elastic_predictor(M, in + i * NIN, d);
    for (int c = 0; c < NOUT; ++c) out[i * NOUT + c] = yn[i * OUT + c] * scale[c] + shift[c] + (c < 6 ? d[c] : 0.0f);
}

// the exact return map in FP32 on physical rows: the method without the network
__global__ void k_exact_fp32(long long n, const float* __restrict__ in, MatConst M, float* __restrict__ out) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float sig[6], e[6];
    for (int c = 0; c < 6; ++c) {
        sig[c] = in[i * NIN + c];
        e[c] = in[i * NIN + 7 + c];
    }
    CrOut<float> o;
    cr_increment<float>(M, in[i * NIN + 6], sig, e, o);
    for (int c = 0; c < 6; ++c) out[i * NOUT + c] = o.dsig[c];
    out[i * NOUT + 6] = o.dR;
}

// the exact return map in FP64 on physical rows, outputs rounded once to
// float (cr_increment_wide); the FP32 form's fallback path computes the same
// map in pairs of floats (cr_increment_pairs)
__global__ void k_exact_wide(long long n, const float* __restrict__ in, MatConst M, float* __restrict__ out) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float sig[6], e[6];
    for (int c = 0; c < 6; ++c) {
        sig[c] = in[i * NIN + c];
        e[c] = in[i * NIN + 7 + c];
    }
    CrOut<double> w;
    cr_increment_wide(M, in[i * NIN + 6], sig, e, w);
    CrOut<float> o;
    cr_narrow(w, o);
    for (int c = 0; c < 6; ++c) out[i * NOUT + c] = o.dsig[c];
    out[i * NOUT + 6] = o.dR;
}

// ---------------------------------------------------------------------------
// BF16 tcgen05 inference (k_mlp_tc, below): tiles of 128 samples; per layer
// one tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, M = 128) per 16 of K with
// the weights (B = W[out][in], N x K) in shared memory, K-major without
// swizzle, and the accumulator D (128 lanes = samples x N columns FP32) in
// tensor memory.  The first layer's A operand (the inputs) is in shared
// memory; the hidden activations are written back to tensor memory
// (tcgen05.st, one lane per sample) and are the A operand of the next layer.
//
// Shared-memory operand layout (K-major, no swizzle): 8-row x 16-byte core
// matrices; element (r, k) of an R-row operand at byte
//   ((k / 8) * (R / 8) + r / 8) * 128 + (r % 8) * 16 + (k % 8) * 2,
// so core matrices adjacent in K are R/8 * 128 bytes apart (the leading
// byte offset) and 8-row groups 128 bytes apart (the stride byte offset).
// ---------------------------------------------------------------------------
__host__ __device__ constexpr uint32_t kmajor_off(int r, int k, int R) {
    return (uint32_t)(((k >> 3) * (R >> 3) + (r >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// shared-memory matrix descriptor: start address, leading and stride byte
// offsets (>> 4), descriptor version 1 (bits 46-47), no swizzle (bits 61-63 = 0)
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// instruction descriptor, kind::f16: D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// shared-memory image of the packed weights (bytes).  The hidden layers'
// biases ride in the MMAs: W1's input column 13 holds b1 (the inputs carry a
// 1 there), and W2, W3 have K = 144 with b2, b3 in column 128 (the
// activations carry a 1 in K column 128, zeros up to 143)
constexpr int KH = HID + 16;
constexpr uint32_t SW1 = 0, SW2 = SW1 + HID * IN * 2, SW3 = SW2 + HID * KH * 2, SW4 = SW3 + HID * KH * 2,
                   WBYTES = SW4 + 16 * HID * 2;  // W4 padded to 16 rows
// biases (FP32): b1, b2, b3 (128 each), b4 (16)
constexpr uint32_t NBIAS = 3 * HID + 16;
// kernel shared memory: weights, biases (FP32; the output bias is used), then
// per tile slot (NSLOT) the inputs A0 (128 x 16), the mbarriers (MMA done and
// final drain per slot), the TMEM address.  Tensor memory per slot (256
// columns): the accumulator D (128 columns), the hidden activations, the A
// operand of layers 2-4 (128 x 144 BF16 = 72 columns, the last 8 the constant
// bias column), so the MMAs read only the weights from shared memory, and the
// last layer's accumulator (16 columns).
constexpr int NSLOT = 2;
constexpr uint32_t SLOT_COLS = 256, TMEM_COLS = SLOT_COLS * NSLOT, ACT_COL = 128, OUT_COL = 208;
constexpr uint32_t S_BIAS = WBYTES, S_A0 = (S_BIAS + NBIAS * 4 + 1023) / 1024 * 1024, A0_BYTES = 128 * IN * 2,
                   S_BAR = S_A0 + NSLOT * A0_BYTES, S_TADDR = S_BAR + 8 * 2 * NSLOT,
                   SMEM_TC = S_TADDR + 8 + 1024;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// one lane of a converged warp (the compiler knows that it is one)
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}

// bounded wait on an mbarrier phase; false (and the error bit) on timeout
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, unsigned* err) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    atomicOr(err, ERR_WAIT_TIMEOUT);
    return false;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// the 32 columns at taddr of this warp's lanes into u, which nothing may use
// before tmem_wait_ld(u)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* u) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
        "%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
          "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]),
          "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
          "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(taddr)
        : "memory");
}

// the load into u (32 words) is done; u passes through, so that no use of it comes before
__device__ __forceinline__ void tmem_wait_ld(uint32_t* u) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 32; ++k) asm volatile("" : "+r"(u[k]));
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

// 16 words of this warp's lanes to TMEM columns taddr .. taddr + 15 (the
// caller waits with tcgen05.wait::st before the columns are read)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* w) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
            taddr),
        "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
        "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
        : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* w) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(w[0]),
                 "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// D (TMEM) = A (TMEM: 128 lanes = rows, two BF16 of K per 32-bit column) x
// B (shared-memory descriptor), accumulate when acc != 0
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc,
                                            uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// ReLU of two accumulators (their biases already summed in), rounded to BF16
// once: v0 to the low half (element k), v1 to the high half
__device__ __forceinline__ uint32_t relu_bf16x2(float v0, float v1) {
    uint32_t y;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(y) : "f"(v1), "f"(v0));
    return y;
}

// issue one layer: D = A (128 x K) . W^T (W: N x K), K in steps of 16
// (the descriptors of successive K steps differ only in the start address
// field, by two core matrices' leading offsets: one addition each)
// with the activations in tensor memory: K / 16 steps of 8 columns
template <int K, int N>
__device__ __forceinline__ void issue_layer_ts(uint32_t tmem, uint32_t a_tmem, uint32_t w_addr) {
    constexpr uint32_t lbo_b = (uint32_t)(N / 8) * 128;
    constexpr uint32_t id = idesc_bf16(128, N);
    uint64_t b = smem_desc(w_addr, lbo_b, 128);
#pragma unroll
    for (int k = 0; k < K; k += 16) {
        mma_bf16_ts(tmem, a_tmem + (uint32_t)(k / 2), b, id, k > 0 ? 1u : 0u);
        b += (2 * lbo_b) >> 4;
    }
}

template <int K, int N>
__device__ __forceinline__ void issue_layer(uint32_t tmem, uint32_t a_addr, uint32_t w_addr) {
    constexpr uint32_t lbo_a = 128 / 8 * 128, lbo_b = (uint32_t)(N / 8) * 128;
    constexpr uint32_t id = idesc_bf16(128, N);
    uint64_t a = smem_desc(a_addr, lbo_a, 128), b = smem_desc(w_addr, lbo_b, 128);
#pragma unroll
    for (int k = 0; k < K; k += 16) {
        mma_bf16(tmem, a, b, id, k > 0 ? 1u : 0u);
        a += (2 * lbo_a) >> 4;
        b += (2 * lbo_b) >> 4;
    }
}

// hidden-layer epilogue of one tile by its group of WPS warps: thread t of
// group warp j (TMEM lane quarter j) owns sample r = 32 j + t; 32 accumulator
// columns at a time it reads them (the bias is in the sums), applies ReLU and
// stores the 16 BF16 pairs to the activation columns of its lane; each load
// runs under the conversions before it
constexpr int WPS = 4;  // epilogue warps per tile slot

__device__ __forceinline__ void relu_store16(uint32_t act_row, const uint32_t* u) {
    uint32_t y[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) y[k] = relu_bf16x2(__uint_as_float(u[2 * k]), __uint_as_float(u[2 * k + 1]));
    tmem_st16(act_row, y);
}

__device__ __forceinline__ void hidden_epilogue(uint32_t d_row, uint32_t act_row) {
    uint32_t u[32], v[32];
    tmem_ld32(d_row, u);
    tmem_wait_ld(u);
    tmem_ld32(d_row + 32u, v);
    relu_store16(act_row, u);
    tmem_wait_ld(v);
    tmem_ld32(d_row + 64u, u);
    relu_store16(act_row + 16u, v);
    tmem_wait_ld(u);
    tmem_ld32(d_row + 96u, v);
    relu_store16(act_row + 32u, u);
    tmem_wait_ld(v);
    relu_store16(act_row + 48u, v);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// a sample's 13 physical inputs (zero past n)
__device__ __forceinline__ void load_inputs(const float* __restrict__ in, long long i, long long n, float x[NIN]) {
#pragma unroll
    for (int c = 0; c < NIN; ++c) x[c] = i < n ? in[i * NIN + c] : 0.0f;
}

// A slot's group and its MMA warp meet when the operand is written and the
// accumulators are read.  True when every thread brings ok, the same answer for
// all, so that after a timeout all of them leave together.
__device__ __forceinline__ bool slot_ready(int slot, bool ok) {
    uint32_t all;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.and.pred.aligned q, %2, %3, p;\n"
        " selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(all)
        : "r"((uint32_t)ok), "r"(1 + slot), "n"(32 * (WPS + 1))
        : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return all != 0u;
}
// the group's side (in_shared: an operand in shared memory, too)
__device__ __forceinline__ bool operand_ready(int slot, bool ok, bool in_shared) {
    if (in_shared) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    return slot_ready(slot, ok);
}

// a warp waits (bounded) for its slot's MMAs; false on a timeout (same answer in every lane)
__device__ __forceinline__ bool group_wait(uint32_t bar, uint32_t parity, unsigned* err) {
    const bool ok = __all_sync(FULL_MASK, bar_wait(bar, parity, err));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return ok;
}

struct TcArgs {
    const uint4* wpack;        // WBYTES of packed BF16 weights (the shared-memory image)
    const float* bias;         // NBIAS
    float in_inv_scale[NIN];
    float out_scale[NOUT], out_shift[NOUT];
    const float* in;           // n x 13 physical
    float* out;                // n x 7 physical
    const unsigned* count;     // device sample count (queue), or null
    long long n;               // sample count (or queue capacity)
    unsigned* err;
    MatConst mat;              // for the elastic predictor D de
};

// row r of a tile's first operand (128 x 16 BF16): the inputs normalised, a 1 in
// column 13 (the bias)
__device__ __forceinline__ void store_inputs(const TcArgs& a, unsigned char* a0, int r, const float x[NIN]) {
    float xn[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) xn[c] = c < NIN ? x[c] * a.in_inv_scale[c] : (c == NIN ? 1.0f : 0.0f);
    uint4 p0, p1;
    p0.x = pack_bf16(xn[0], xn[1]);
    p0.y = pack_bf16(xn[2], xn[3]);
    p0.z = pack_bf16(xn[4], xn[5]);
    p0.w = pack_bf16(xn[6], xn[7]);
    p1.x = pack_bf16(xn[8], xn[9]);
    p1.y = pack_bf16(xn[10], xn[11]);
    p1.z = pack_bf16(xn[12], xn[13]);
    p1.w = pack_bf16(xn[14], xn[15]);
    *reinterpret_cast<uint4*>(a0 + kmajor_off(r, 0, 128)) = p0;
    *reinterpret_cast<uint4*>(a0 + kmajor_off(r, 8, 128)) = p1;
}

// sample i's outputs from its lane's 16 output columns: the network's correction
// plus the elastic predictor D de, and dR
__device__ __forceinline__ void write_outputs(const TcArgs& a, uint32_t out_row, const float* bias, const float de[6],
                                              long long i, long long n) {
    float v[16];
    tmem_ld16(out_row, v);
    if (i >= n) return;
    float d[6];
    trial_increment<float>(a.mat, de, d);
#pragma unroll
    for (int c = 0; c < NOUT; ++c)
        a.out[i * NOUT + c] = (v[c] + bias[3 * HID + c]) * a.out_scale[c] + a.out_shift[c] + (c < 6 ? d[c] : 0.0f);
}

// NSLOT epilogue groups of WPS warps (one per tile slot; warp j of a group
// reads TMEM lane quarter j) and an MMA warp per slot
constexpr int TC_THREADS = 32 * (WPS + 1) * NSLOT;

// One CTA per SM takes groups of NSLOT 128-sample tiles, one per slot, and
// runs the slots as independent pipelines that share the tensor core.  A
// slot's epilogue group writes the operand (the inputs into shared memory,
// the activations into tensor memory) and meets the slot's MMA warp
// (slot_ready), which issues the layer and commits it to the slot's `full`
// mbarrier; the group waits on `full`, turns the accumulators into the next
// operand, and so on.  A tile has three hand-offs, not four: its fourth layer
// goes with the next tile's first, whose operand is written, and the last
// tile's outputs and the next tile's inputs are dealt with, while the second
// layer runs.
//
// Bound by the MMAs of the two slots, which take turns: 1,432 clocks per tile
// (nine of 64 in each hidden layer, eight of 27 in the last), 2,860 of the
// 3,470 a pair of tiles takes.  8M samples: 372 us, 1.52 PFLOP/s (654 us with
// one MMA warp that issued under a test of its lane number: an MMA takes
// uniform operands, and each one went round a loop over the lanes, 64 to 79
// clocks; elected lanes issue one in 16).  300k samples 33 -> 23.5 us.  Tried:
// the group's first warp issuing (437 us; its own epilogue waits meanwhile), an
// mbarrier in place of slot_ready (376).
// Waits are bounded: on a timeout the error word is set and the roles stop;
// the MMA warps then wait (bounded) for their last MMAs before the TMEM is
// freed.
__global__ void __launch_bounds__(TC_THREADS, 1) k_mlp_tc(TcArgs a) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const int t = threadIdx.x, w = t >> 5;
    unsigned char* s = sm + ((1024 - (smem_u32(sm) & 1023u)) & 1023u);  // 1024-byte aligned base
    const uint32_t sbase = smem_u32(s);
    // weights and biases into shared memory (once per CTA)
    for (uint32_t i = t; i < WBYTES / 16; i += TC_THREADS) reinterpret_cast<uint4*>(s)[i] = a.wpack[i];
    float* bias = reinterpret_cast<float*>(s + S_BIAS);
    for (uint32_t i = t; i < NBIAS; i += TC_THREADS) bias[i] = a.bias[i];
    uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(s + S_TADDR);
    // mbarriers: slot sl's MMA-done at full0 + 8 sl, its operand-ready at ready0 + 8 sl
    const uint32_t full0 = sbase + S_BAR, drain0 = full0 + 8 * NSLOT;
    if (t == 0) {
        for (uint32_t sl = 0; sl < NSLOT; ++sl) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * sl) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(drain0 + 8 * sl) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (w == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(taddr_slot)),
                     "n"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *taddr_slot;
    const long long n = a.count ? (long long)min((unsigned long long)*a.count, (unsigned long long)a.n) : a.n;
    const long long ngroups = (n + 128 * NSLOT - 1) / (128 * NSLOT);
    // tile groups of this CTA: blockIdx.x, blockIdx.x + gridDim.x, ...
    const long long mine = blockIdx.x < ngroups ? (ngroups - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    if (w >= WPS * NSLOT) {
        // slot sl's MMA warp: issues a layer whenever its group has the operand ready
        const int sl = w - WPS * NSLOT;
        const uint32_t full = full0 + 8u * sl;
        const uint32_t d = tmem + SLOT_COLS * sl, act = d + ACT_COL;
        bool ok = mine > 0;
        for (long long k = 0; k < mine; ++k) {
            if (!(ok = slot_ready(sl, true))) break;
            if (elect_one()) {
                if (k > 0) issue_layer_ts<HID, 16>(d + OUT_COL, act, sbase + SW4);  // of the last tile
                issue_layer<IN, HID>(d, sbase + S_A0 + sl * A0_BYTES, sbase + SW1);
                mma_commit(full);
            }
            __syncwarp();
            if (!(ok = slot_ready(sl, true))) break;
            if (elect_one()) {
                issue_layer_ts<KH, HID>(d, act, sbase + SW2);
                mma_commit(full);
            }
            __syncwarp();
            if (!(ok = slot_ready(sl, true))) break;
            if (elect_one()) {
                issue_layer_ts<KH, HID>(d, act, sbase + SW3);
                mma_commit(full);
            }
            __syncwarp();
        }
        if (ok && slot_ready(sl, true)) {
            if (elect_one()) {
                issue_layer_ts<HID, 16>(d + OUT_COL, act, sbase + SW4);
                mma_commit(full);
            }
            __syncwarp();
        }
        // every MMA issued has completed before the TMEM is freed
        if (elect_one()) {
            mma_commit(drain0 + 8u * sl);
            bar_wait(drain0 + 8u * sl, 0u, a.err);
        }
        __syncwarp();
    } else {
        // epilogue group = slot sl; its warp j reads lanes 32 j .. + 31, one sample per lane
        const int sl = w / WPS, j = w % WPS, r = 32 * j + (t & 31);
        const uint32_t full = full0 + 8u * sl;
        const uint32_t trow = tmem + SLOT_COLS * (uint32_t)sl + ((uint32_t)(32 * j) << 16);
        unsigned char* a0 = s + S_A0 + sl * A0_BYTES;
        {
            // the activations' constant K columns 128 .. 143: 1, 0, ..., 0 (the bias column)
            uint32_t one[8] = {0x3F80u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            tmem_st8(trow + ACT_COL + HID / 2, one);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        const long long stride = (long long)gridDim.x * NSLOT * 128;
        long long i = ((long long)blockIdx.x * NSLOT + sl) * 128 + r;  // this tile's sample
        uint32_t ph = 0u;
        bool ok = mine > 0;
        float x[NIN], de[6], de_out[6];  // the next tile's physical inputs; strain increments of this tile and the last
        load_inputs(a.in, i, n, x);
        store_inputs(a, a0, r, x);
#pragma unroll
        for (int c = 0; c < 6; ++c) de[c] = de_out[c] = x[7 + c];
        if (ok) ok = operand_ready(sl, true, true);
        load_inputs(a.in, i + stride, n, x);
        for (long long k = 0; k < mine && ok; ++k) {
            // first layer done (and the last tile's outputs)
            ok = group_wait(full, ph, a.err);
            if (ok) hidden_epilogue(trow, trow + ACT_COL);
            if (!(ok = operand_ready(sl, ok, false))) break;
            // while the second runs: the last tile's outputs, the next tile's operand
            if (k > 0) write_outputs(a, trow + OUT_COL, bias, de_out, i - stride, n);
            store_inputs(a, a0, r, x);
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                de_out[c] = de[c];
                de[c] = x[7 + c];
            }
            load_inputs(a.in, i + 2 * stride, n, x);
            ok = group_wait(full, ph ^ 1u, a.err);
            if (ok) hidden_epilogue(trow, trow + ACT_COL);
            if (!(ok = operand_ready(sl, ok, false))) break;
            ok = group_wait(full, ph, a.err);
            if (ok) hidden_epilogue(trow, trow + ACT_COL);
            ok = operand_ready(sl, ok, true);  // and the next tile's inputs
            ph ^= 1u;
            i += stride;
        }
        if (ok && group_wait(full, ph, a.err)) write_outputs(a, trow + OUT_COL, bias, de_out, i - stride, n);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (w == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
}

}  // namespace net
}  // namespace mpm

using namespace mpm;
using namespace mpm::net;

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct mpm_net {
    mpm_net_config cfg;
    MatConst mat;
    int sm_count = 152;
    float* p = nullptr;      // NPARAM master parameters
    float* wpack = nullptr;  // packed BF16 weight image (WBYTES) + biases (NBIAS floats)
    float* scratch = nullptr;
    size_t scratch_bytes = 0;
    unsigned* err = nullptr;
    void* h_result = nullptr;  // pinned: mpm_net_loss_grad's gradient and loss
    float in_inv_scale[NIN];
    float out_scale[NOUT], out_shift[NOUT];
    bool packed = false;
    // box of the normalised training inputs (the guard's first check); unbounded until trained
    float box_lo[NIN], box_hi[NIN];
};

static MatConst make_mat(const mpm_net_config& c) {
    MatConst k;
    memset(&k, 0, sizeof(k));
    const double E = c.E, nu = c.nu;
    k.type = 4;
    k.E = E;
    k.nu = nu;
    k.Y = c.yield;
    k.C0 = c.C0;
    k.C1 = c.C1;
    k.C = E / (1.0 + nu) / (1.0 - 2.0 * nu);
    k.one_m_nu = 1.0 - nu;
    k.half_m_nu = 0.5 - nu;
    k.G = 0.5 * E / (1.0 + nu);
    k.k0 = c.yield / std::sqrt(3.0);
    k.s23C1 = std::sqrt(2.0 / 3.0) * c.C1;
    k.inv_E = 1.0 / E;
    k.nu_over_E = nu / E;
    k.inv_G = 1.0 / k.G;
    set_float_constants(k);
    return k;
}

static int ensure_scratch(mpm_net* net, size_t bytes) {
    if (net->scratch_bytes >= bytes) return MPM_OK;
    if (net->scratch) cudaFree(net->scratch);
    net->scratch = nullptr;
    net->scratch_bytes = 0;
    if (cudaMalloc(&net->scratch, bytes) != cudaSuccess) {
        cudaGetLastError();
        return MPM_ERR_NOMEM;
    }
    net->scratch_bytes = bytes;
    return MPM_OK;
}

// BF16 image of the weights in the inference kernel's shared-memory layout
static int pack_weights(mpm_net* net) {
    std::vector<float> p(NPARAM);
    NCK(cudaMemcpy(p.data(), net->p, NPARAM * 4, cudaMemcpyDeviceToHost));
    std::vector<uint16_t> img(WBYTES / 2, 0);
    auto bf = [](float f) -> uint16_t {
        uint32_t u;
        memcpy(&u, &f, 4);
        if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)((u >> 16) | 0x40u);
        u += 0x7fffu + ((u >> 16) & 1u);
        return (uint16_t)(u >> 16);
    };
    // R x Kimg image of the R x K weights at off, the bias at boff in column kb (kb < 0: none)
    auto put = [&](uint32_t base, int R, int K, int Kimg, long long off, int rows_valid, int kb, long long boff) {
        for (int r = 0; r < R; ++r)
            for (int k = 0; k < Kimg; ++k) {
                float v = 0.0f;
                if (r < rows_valid && k == kb) v = p[boff + r];
                else if (r < rows_valid && k < K) v = p[off + (long long)r * K + k];
                img[(base + kmajor_off(r, k, R)) / 2] = bf(v);
            }
    };
    put(SW1, HID, IN, IN, OW1, HID, NIN, OB1);
    put(SW2, HID, HID, KH, OW2, HID, HID, OB2);
    put(SW3, HID, HID, KH, OW3, HID, HID, OB3);
    put(SW4, 16, HID, HID, OW4, OUT, -1, 0);
    std::vector<float> bias(NBIAS, 0.0f);
    for (int i = 0; i < HID; ++i) {
        bias[i] = p[OB1 + i];
        bias[HID + i] = p[OB2 + i];
        bias[2 * HID + i] = p[OB3 + i];
    }
    for (int i = 0; i < OUT; ++i) bias[3 * HID + i] = p[OB4 + i];
    if (!net->wpack && cudaMalloc(&net->wpack, WBYTES + NBIAS * 4) != cudaSuccess) {
        cudaGetLastError();
        return MPM_ERR_NOMEM;
    }
    NCK(cudaMemcpy(net->wpack, img.data(), WBYTES, cudaMemcpyHostToDevice));
    NCK(cudaMemcpy((char*)net->wpack + WBYTES, bias.data(), NBIAS * 4, cudaMemcpyHostToDevice));
    net->packed = true;
    return MPM_OK;
}

// the hidden layers on normalised rows x (n x 16): h1..h3 (n x 128 each)
static void hidden_fp32(mpm_net* net, cudaStream_t s, long long n, const float* x, float* h1, float* h2, float* h3) {
    const float* p = net->p;
    const float* none = nullptr;
    float* no_sums = nullptr;
    const long long tiles = (n + 127) / 128;
    launch_net(s, k_layer<true, IN>, tiles, GT, sizeof(GemmTile), (int)n, x, p + OW1, p + OB1, none, h1, no_sums);
    launch_net(s, k_layer<true, HID>, tiles, GT, sizeof(GemmTile), (int)n, (const float*)h1, p + OW2, p + OB2, none, h2,
               no_sums);
    launch_net(s, k_layer<true, HID>, tiles, GT, sizeof(GemmTile), (int)n, (const float*)h2, p + OW3, p + OB3, none, h3,
               no_sums);
}

static long long head_blocks(const mpm_net* net, long long n) {
    return std::max(1LL, std::min<long long>(net->sm_count, (n + HEAD_WARPS - 1) / HEAD_WARPS));
}

// forward pass on normalised rows x; y (n x 8)
static void forward_fp32(mpm_net* net, cudaStream_t s, long long n, const float* x, float* h1, float* h2, float* h3,
                         float* y) {
    hidden_fp32(net, s, n, x, h1, h2, h3);
    const float* p = net->p;
    launch_net(s, k_head<false>, head_blocks(net, n) * 2, HEAD_WARPS * 32, 0, n, (const float*)h3, p + OW4, p + OB4,
               (const float*)nullptr, y, (float*)nullptr, (float*)nullptr, (float*)nullptr, (float*)nullptr,
               (double*)nullptr);
}

// loss (added to *loss) and its gradient into g (NPARAM, zeroed here) on rows x, t; h1..h3, da, db scratch (n x 128)
static void loss_grad_fp32(mpm_net* net, cudaStream_t s, long long n, const float* x, const float* t, float* h1,
                           float* h2, float* h3, float* da, float* db, float* g, double* loss) {
    const float* p = net->p;
    const float* none = nullptr;
    cudaMemsetAsync(g, 0, NPARAM * 4, s);
    hidden_fp32(net, s, n, x, h1, h2, h3);
    launch_net(s, k_head<true>, head_blocks(net, n), HEAD_WARPS * 32, 0, n, (const float*)h3, p + OW4, p + OB4, t,
               (float*)nullptr, da, g + OW4, g + OB4, g + OB3, loss);
    // the weight gradients' rows over two blocks per SM, whole slices each
    const long long blocks = 2LL * net->sm_count;
    const int rows = (int)(((n + blocks - 1) / blocks + GK - 1) / GK * GK);
    const long long wb = (n + rows - 1) / rows, tiles = (n + 127) / 128;
    const size_t sm = sizeof(GemmTile);
    launch_net(s, k_weight_grad<HID>, wb, GT, sm, (int)n, rows, (const float*)da, (const float*)h2, g + OW3);
    launch_net(s, k_layer<false, HID>, tiles, GT, sm, (int)n, (const float*)da, p + OW3, none, (const float*)h2, db,
               g + OB2);
    launch_net(s, k_weight_grad<HID>, wb, GT, sm, (int)n, rows, (const float*)db, (const float*)h1, g + OW2);
    launch_net(s, k_layer<false, HID>, tiles, GT, sm, (int)n, (const float*)db, p + OW2, none, (const float*)h1, da,
               g + OB1);
    launch_net(s, k_weight_grad<IN>, wb, GT, sm, (int)n, rows, (const float*)da, x, g + OW1);
}

extern "C" {

int64_t mpm_net_param_count(void) { return NPARAM; }

int mpm_net_create(const mpm_net_config* cfg, mpm_net** out) {
    if (!cfg || !out) return MPM_ERR_ARG;
    *out = nullptr;
    if (!(cfg->E > 0) || !(cfg->nu > -1.0 && cfg->nu < 0.5) || !(cfg->yield > 0) || cfg->n_samples < 1 ||
        cfg->batch < 64 || cfg->epochs < 0 || !(cfg->deps_sigma > 0) || !(cfg->stress_range > 0) ||
        (cfg->sampling != 0 && cfg->sampling != 1))
        return MPM_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return MPM_ERR_CUDA;
    }
    mpm_net* net = new (std::nothrow) mpm_net();
    if (!net) return MPM_ERR_NOMEM;
    net->cfg = *cfg;
    net->mat = make_mat(*cfg);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&net->sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (cudaMalloc(&net->p, NPARAM * 4) != cudaSuccess || cudaMalloc(&net->err, 4) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_TC) != cudaSuccess) {
        cudaGetLastError();
        mpm_net_destroy(net);
        return MPM_ERR_NOMEM;
    }
    cudaMemset(net->err, 0, 4);
    // initial parameters: U(-1/sqrt(fan_in), 1/sqrt(fan_in)) (padded input columns zero)
    std::vector<float> p(NPARAM, 0.0f);
    uint64_t st = cfg->seed * 0x2545F4914F6CDD1DULL + 12345;
    auto u = [&]() {
        st += 0x9e3779b97f4a7c15ULL;
        return (double)(mix64(st) >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    for (int r = 0; r < HID; ++r)
        for (int k = 0; k < NIN; ++k) p[OW1 + r * IN + k] = (float)(u() / std::sqrt((double)NIN));
    for (int r = 0; r < HID; ++r) p[OB1 + r] = (float)(u() / std::sqrt((double)NIN));
    for (long long i = 0; i < HID * HID; ++i) p[OW2 + i] = (float)(u() / std::sqrt((double)HID));
    for (int r = 0; r < HID; ++r) p[OB2 + r] = (float)(u() / std::sqrt((double)HID));
    for (long long i = 0; i < HID * HID; ++i) p[OW3 + i] = (float)(u() / std::sqrt((double)HID));
    for (int r = 0; r < HID; ++r) p[OB3 + r] = (float)(u() / std::sqrt((double)HID));
    for (long long i = 0; i < OUT * HID; ++i) p[OW4 + i] = i < NOUT * HID ? (float)(u() / std::sqrt((double)HID)) : 0.0f;
    for (int r = 0; r < NOUT; ++r) p[OB4 + r] = (float)(u() / std::sqrt((double)HID));
    if (cudaMemcpy(net->p, p.data(), NPARAM * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        mpm_net_destroy(net);
        return MPM_ERR_CUDA;
    }
    for (int c = 0; c < 6; ++c) {
        net->in_inv_scale[c] = (float)(1.0 / cfg->yield);
        net->in_inv_scale[7 + c] = (float)(1.0 / cfg->deps_sigma);
    }
    net->in_inv_scale[6] = (float)(1.0 / cfg->yield);
    for (int c = 0; c < NIN; ++c) {
        net->box_lo[c] = -INFINITY;
        net->box_hi[c] = INFINITY;
    }
    for (int c = 0; c < NOUT; ++c) {
        net->out_scale[c] = 1.0f;
        net->out_shift[c] = 0.0f;
    }
    *out = net;
    return MPM_OK;
}

void mpm_net_destroy(mpm_net* net) {
    if (!net) return;
    if (net->p) cudaFree(net->p);
    if (net->wpack) cudaFree(net->wpack);
    if (net->scratch) cudaFree(net->scratch);
    if (net->err) cudaFree(net->err);
    if (net->h_result) cudaFreeHost(net->h_result);
    delete net;
}

int mpm_net_get_params(mpm_net* net, float* host, int64_t n) {
    if (!net || !host || n != NPARAM) return MPM_ERR_ARG;
    NCK(cudaMemcpy(host, net->p, NPARAM * 4, cudaMemcpyDeviceToHost));
    return MPM_OK;
}

int mpm_net_set_params(mpm_net* net, const float* host, int64_t n) {
    if (!net || !host || n != NPARAM) return MPM_ERR_ARG;
    NCK(cudaMemcpy(net->p, host, NPARAM * 4, cudaMemcpyHostToDevice));
    return pack_weights(net);
}

int mpm_net_scales(mpm_net* net, double in_scale[13], double out_scale[7], double out_shift[7]) {
    if (!net) return MPM_ERR_ARG;
    for (int c = 0; c < NIN; ++c)
        if (in_scale) in_scale[c] = 1.0 / (double)net->in_inv_scale[c];
    for (int c = 0; c < NOUT; ++c) {
        if (out_scale) out_scale[c] = net->out_scale[c];
        if (out_shift) out_shift[c] = net->out_shift[c];
    }
    return MPM_OK;
}

int mpm_net_loss_grad(mpm_net* net, const float* x, const float* t, int64_t n, float* grad, double* loss) {
    if (!net || !x || !t || !grad || n < 1) return MPM_ERR_ARG;
    const size_t need = 4 * ((size_t)n * (IN + OUT) + (size_t)n * HID * 5 + NPARAM) + 64;
    int rc = ensure_scratch(net, need);
    if (rc) return rc;
    // gradient and loss come back in one copy, through a pinned buffer
    constexpr size_t RESULT = (NPARAM * 4 + 15) / 16 * 16 + 8;
    if (!net->h_result && cudaMallocHost(&net->h_result, RESULT) != cudaSuccess) {
        cudaGetLastError();
        net->h_result = nullptr;
        return MPM_ERR_NOMEM;
    }
    float* xs = net->scratch;
    float* ts = xs + n * IN;
    float* h1 = ts + n * OUT;
    float* h2 = h1 + n * HID;
    float* h3 = h2 + n * HID;
    float* d1 = h3 + n * HID;
    float* d2 = d1 + n * HID;
    float* g = d2 + n * HID;
    double* dl = reinterpret_cast<double*>(g + (RESULT - 8) / 4);
    cudaStream_t s = 0;
    NCK(cudaMemcpy(xs, x, (size_t)n * IN * 4, cudaMemcpyHostToDevice));
    NCK(cudaMemcpy(ts, t, (size_t)n * OUT * 4, cudaMemcpyHostToDevice));
    NCK(cudaMemsetAsync(dl, 0, 8, s));
    loss_grad_fp32(net, s, n, xs, ts, h1, h2, h3, d1, d2, g, dl);
    NCK(cudaGetLastError());
    NCK(cudaMemcpyAsync(net->h_result, g, RESULT, cudaMemcpyDeviceToHost, s));
    NCK(cudaStreamSynchronize(s));
    memcpy(grad, net->h_result, NPARAM * 4);
    if (loss) memcpy(loss, (const char*)net->h_result + RESULT - 8, 8);
    return MPM_OK;
}

static int train_impl(mpm_net* net, const float* d_rows, long long n_rows, mpm_net_report* rep) {
    const mpm_net_config& c = net->cfg;
    const long long nval = d_rows ? std::max(1LL, std::min(65536LL, n_rows / 20)) : std::max(65536LL, (long long)c.n_samples / 100);
    const long long n = d_rows ? n_rows - nval : (long long)c.n_samples, B = std::min<long long>(c.batch, n);
    if (n < 64) return MPM_ERR_ARG;
    mpm_net_report r;
    memset(&r, 0, sizeof(r));
    // data: x (n x 16), t (n x 8 physical), tn (n x 8 normalised), raw inputs (n x 13)
    float *x = nullptr, *t = nullptr, *tn = nullptr, *xv = nullptr, *tv = nullptr;
    auto freeall = [&]() {
        for (float* q : {x, t, tn, xv, tv})
            if (q) cudaFree(q);
    };
    if (cudaMalloc(&x, (size_t)n * IN * 4) != cudaSuccess || cudaMalloc(&t, (size_t)n * OUT * 4) != cudaSuccess ||
        cudaMalloc(&tn, (size_t)n * OUT * 4) != cudaSuccess || cudaMalloc(&xv, (size_t)nval * IN * 4) != cudaSuccess ||
        cudaMalloc(&tv, (size_t)nval * OUT * 4) != cudaSuccess) {
        cudaGetLastError();
        freeall();
        return MPM_ERR_NOMEM;
    }
    SampleCfg sc{c.yield, c.stress_range, c.epbar_max, c.deps_sigma, c.C0, c.C1, c.seed, c.sampling};
    auto t0 = std::chrono::steady_clock::now();
    if (d_rows) {
        k_label_rows<<<(unsigned)((n + 255) / 256), 256>>>(n, d_rows, sc, net->mat, x, t);
        k_label_rows<<<(unsigned)((nval + 255) / 256), 256>>>(nval, d_rows + n * NIN, sc, net->mat, xv, tv);
    } else {
        k_generate<<<(unsigned)((n + 255) / 256), 256>>>(n, 0, sc, net->mat, x, t);
        k_generate<<<(unsigned)((nval + 255) / 256), 256>>>(nval, n, sc, net->mat, xv, tv);
    }
    // output normalisation from the training set
    double* acc = nullptr;
    float* dvec = nullptr;
    if (cudaMalloc(&acc, 64 * 8) != cudaSuccess || cudaMalloc(&dvec, 64 * 4) != cudaSuccess) {
        cudaGetLastError();
        freeall();
        return MPM_ERR_NOMEM;
    }
    {  // the box of the training inputs, for the guard
        unsigned hb[2 * NIN];
        for (int c = 0; c < NIN; ++c) {
            hb[c] = 0xffffffffu;
            hb[NIN + c] = 0u;
        }
        unsigned* db = reinterpret_cast<unsigned*>(dvec);
        cudaMemcpy(db, hb, sizeof(hb), cudaMemcpyHostToDevice);
        k_box<<<net->sm_count * 4, 256>>>(n, x, db);
        cudaMemcpy(hb, db, sizeof(hb), cudaMemcpyDeviceToHost);
        for (int c = 0; c < NIN; ++c) {
            net->box_lo[c] = ord2f(hb[c]);
            net->box_hi[c] = ord2f(hb[NIN + c]);
        }
    }
    cudaMemset(acc, 0, 64 * 8);
    k_moments<<<net->sm_count * 4, 256>>>(n, t, acc);
    double h[2 * NOUT];
    cudaMemcpy(h, acc, sizeof(h), cudaMemcpyDeviceToHost);
    float fs[2 * NOUT];
    for (int k = 0; k < NOUT; ++k) {
        const double mean = h[k] / n, var = std::max(h[NOUT + k] / n - mean * mean, 1e-30);
        net->out_shift[k] = (float)mean;
        net->out_scale[k] = (float)std::sqrt(var);
        fs[k] = net->out_shift[k];
        fs[NOUT + k] = 1.0f / net->out_scale[k];
        r.out_shift[k] = net->out_shift[k];
        r.out_scale[k] = net->out_scale[k];
    }
    cudaMemcpy(dvec, fs, sizeof(fs), cudaMemcpyHostToDevice);
    k_normalise_targets<<<(unsigned)((n + 255) / 256), 256>>>(n, t, dvec, dvec + NOUT, tn);
    if (cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        freeall();
        cudaFree(acc);
        cudaFree(dvec);
        return MPM_ERR_CUDA;
    }
    auto t1 = std::chrono::steady_clock::now();
    r.seconds_generate = std::chrono::duration<double>(t1 - t0).count();
    // training buffers
    const size_t need = 4 * ((size_t)B * (IN + 2 * OUT) + (size_t)B * HID * 5 + 3 * NPARAM) + 1024;
    int rc = ensure_scratch(net, need);
    if (rc) {
        freeall();
        cudaFree(acc);
        cudaFree(dvec);
        return rc;
    }
    float* xb = net->scratch;
    float* tb = xb + B * IN;
    float* y = tb + B * OUT;
    float* h1 = y + B * OUT;
    float* h2 = h1 + B * HID;
    float* h3 = h2 + B * HID;
    float* d1 = h3 + B * HID;
    float* d2 = d1 + B * HID;
    float* g = d2 + B * HID;
    float* m1 = g + NPARAM;
    float* m2 = m1 + NPARAM;
    cudaMemset(m1, 0, 2 * NPARAM * 4);
    const long long per_epoch = n / B;
    const long long total = per_epoch * c.epochs;
    static const long long primes[] = {1000003, 2750159, 4256249, 7368787, 9999991, 15485863, 32452843,
                                       49979687, 67867967, 86028121, 104395301, 122949823};
    long long step = 0;
    cudaStream_t s = 0;
    for (int ep = 0; ep < c.epochs; ++ep) {
        long long a = primes[ep % 12];
        while (std::gcd(a, n) != 1) a += 2;
        const long long cc = (long long)(mix64(c.seed + ep) % (uint64_t)n);
        cudaMemsetAsync(acc + 32, 0, 8, s);
        for (long long b = 0; b < per_epoch; ++b, ++step) {
            k_gather<<<(unsigned)((B + 255) / 256), 256, 0, s>>>(n, x, tn, a, cc, b * B, (int)B, xb, tb);
            loss_grad_fp32(net, s, B, xb, tb, h1, h2, h3, d1, d2, g, acc + 32);
            // Adam, cosine-decayed step size after a short warm-up
            const double tt = (double)(step + 1);
            const double warm = std::min(1.0, tt / (double)std::max(1LL, std::min(200LL, total / 10)));
            const double lr = c.lr * warm * (0.02 + 0.98 * 0.5 * (1.0 + std::cos(3.14159265358979323846 * (double)step / (double)total)));
            const float c1 = (float)(1.0 - std::pow(0.9, tt)), c2 = (float)(1.0 - std::pow(0.999, tt));
            k_adam<<<(unsigned)((NPARAM + 255) / 256), 256, 0, s>>>(NPARAM, net->p, g, m1, m2, (float)lr, 0.9f, 0.999f,
                                                                    1e-8f, c1, c2);
        }
        double lsum = 0.0;
        cudaMemcpy(&lsum, acc + 32, 8, cudaMemcpyDeviceToHost);
        const double lmean = per_epoch ? lsum / per_epoch : 0.0;
        if (ep == 0) r.loss_first = lmean;
        r.loss_last = lmean;
    }
    if (cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        freeall();
        cudaFree(acc);
        cudaFree(dvec);
        return MPM_ERR_CUDA;
    }
    auto t2 = std::chrono::steady_clock::now();
    r.seconds_train = std::chrono::duration<double>(t2 - t1).count();
    r.steps = step;
    // held-out errors with the FP32 forward pass
    rc = MPM_OK;
    {
        const long long chunk = std::min(nval, B);
        float fsh[2 * NOUT];
        for (int k = 0; k < NOUT; ++k) {
            fsh[k] = net->out_shift[k];
            fsh[NOUT + k] = net->out_scale[k];
        }
        cudaMemcpy(dvec, fsh, sizeof(fsh), cudaMemcpyHostToDevice);
        cudaMemset(acc, 0, 16 * 8);
        unsigned* maxbits = reinterpret_cast<unsigned*>(acc + 8);
        for (long long o = 0; o < nval; o += chunk) {
            const long long m = std::min(chunk, nval - o);
            forward_fp32(net, s, m, xv + o * IN, h1, h2, h3, y);
            k_val_errors<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(m, y, tv + o * OUT, dvec, dvec + NOUT,
                                                                    (float)(1.0 / c.yield), 0.02f, acc, maxbits);
        }
        double v[4];
        unsigned mb = 0;
        cudaMemcpy(v, acc, sizeof(v), cudaMemcpyDeviceToHost);
        cudaMemcpy(&mb, maxbits, 4, cudaMemcpyDeviceToHost);
        float mx;
        memcpy(&mx, &mb, 4);
        r.n_val = nval;
        r.val_rms_dsig = std::sqrt(v[0] / (6.0 * nval));
        r.val_rms_dsig_outside = v[3] > 0 ? std::sqrt(v[1] / (6.0 * v[3])) : 0.0;
        r.val_max_dsig = mx;
        r.val_rms_dR = std::sqrt(v[2] / nval);
        if (cudaDeviceSynchronize() != cudaSuccess) {
            cudaGetLastError();
            rc = MPM_ERR_CUDA;
        }
    }
    freeall();
    cudaFree(acc);
    cudaFree(dvec);
    if (rc) return rc;
    rc = pack_weights(net);
    if (rep) *rep = r;
    return rc;
}

int mpm_net_train(mpm_net* net, mpm_net_report* rep) {
    if (!net) return MPM_ERR_ARG;
    return train_impl(net, nullptr, 0, rep);
}

int mpm_net_train_rows(mpm_net* net, const float* d_rows, int64_t n, mpm_net_report* rep) {
    if (!net || !d_rows || n < 128) return MPM_ERR_ARG;
    return train_impl(net, d_rows, n, rep);
}

int mpm_net_infer(mpm_net* net, const float* d_in, float* d_out, int64_t n, int kernel, void* stream) {
    if (!net || n < 0 || kernel < 0 || kernel > 3) return MPM_ERR_ARG;
    if (n == 0) return MPM_OK;
    if (!d_in || !d_out) return MPM_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (kernel == 2) {
        k_exact_fp32<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, d_in, net->mat, d_out);
        NCK(cudaGetLastError());
        return MPM_OK;
    }
    if (kernel == 3) {
        k_exact_wide<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, d_in, net->mat, d_out);
        NCK(cudaGetLastError());
        return MPM_OK;
    }
    if (!net->packed) {
        int rc = pack_weights(net);
        if (rc) return rc;
    }
    if (kernel == 0) {
        TcArgs a;
        a.wpack = reinterpret_cast<const uint4*>(net->wpack);
        a.bias = reinterpret_cast<const float*>((const char*)net->wpack + WBYTES);
        for (int c = 0; c < NIN; ++c) a.in_inv_scale[c] = net->in_inv_scale[c];
        for (int c = 0; c < NOUT; ++c) {
            a.out_scale[c] = net->out_scale[c];
            a.out_shift[c] = net->out_shift[c];
        }
        a.in = d_in;
        a.out = d_out;
        a.count = nullptr;
        a.n = n;
        a.err = net->err;
        a.mat = net->mat;
        const long long groups = (n + 128 * NSLOT - 1) / (128 * NSLOT);
        const unsigned grid = (unsigned)std::min<long long>(std::max<long long>(groups, 1), net->sm_count);
        k_mlp_tc<<<grid, TC_THREADS, SMEM_TC, s>>>(a);
        NCK(cudaGetLastError());
        return MPM_OK;
    }
    // FP32 reference: normalise, the training forward pass in chunks, de-normalise
    const long long chunk = std::min<long long>(n, 1 << 20);
    const size_t need = 4 * ((size_t)chunk * (IN + OUT) + (size_t)chunk * HID * 3 + 2 * NIN + 2 * NOUT) + 256;
    int rc = ensure_scratch(net, need);
    if (rc) return rc;
    float* x = net->scratch;
    float* y = x + chunk * IN;
    float* h1 = y + chunk * OUT;
    float* h2 = h1 + chunk * HID;
    float* h3 = h2 + chunk * HID;
    float* sc = h3 + chunk * HID;
    float hs[NIN + 2 * NOUT];
    for (int c = 0; c < NIN; ++c) hs[c] = net->in_inv_scale[c];
    for (int c = 0; c < NOUT; ++c) {
        hs[NIN + c] = net->out_scale[c];
        hs[NIN + NOUT + c] = net->out_shift[c];
    }
    NCK(cudaMemcpyAsync(sc, hs, sizeof(hs), cudaMemcpyHostToDevice, s));
    for (long long o = 0; o < n; o += chunk) {
        const long long m = std::min(chunk, n - o);
        k_norm_inputs<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(m, d_in + o * NIN, sc, x);
        forward_fp32(net, s, m, x, h1, h2, h3, y);
        k_denorm_outputs<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(m, y, sc + NIN, sc + NIN + NOUT,
                                                                     d_in + o * NIN, net->mat, d_out + o * NOUT);
    }
    NCK(cudaStreamSynchronize(s));
    return MPM_OK;
}

}  // extern "C"

namespace mpm {
int net_run_queue(mpm_net* net, const SurrogateQueue& q, cudaStream_t s, unsigned* err) {
    if (!net->packed) {
        int rc = pack_weights(net);
        if (rc) return rc;
    }
    TcArgs a;
    a.wpack = reinterpret_cast<const uint4*>(net->wpack);
    a.bias = reinterpret_cast<const float*>((const char*)net->wpack + WBYTES);
    for (int c = 0; c < NIN; ++c) a.in_inv_scale[c] = net->in_inv_scale[c];
    for (int c = 0; c < NOUT; ++c) {
        a.out_scale[c] = net->out_scale[c];
        a.out_shift[c] = net->out_shift[c];
    }
    a.in = q.in;
    a.out = q.out;
    a.count = q.count;
    a.n = q.cap;
    a.err = err;
    a.mat = net->mat;
    k_mlp_tc<<<(unsigned)net->sm_count, TC_THREADS, SMEM_TC, s>>>(a);
    return cudaGetLastError() == cudaSuccess ? MPM_OK : MPM_ERR_CUDA;
}

float net_yield(const mpm_net* net) { return (float)net->cfg.yield; }
SurrogateGuard net_guard(const mpm_net* net, float tol) {
    SurrogateGuard g;
    for (int c = 0; c < NIN; ++c) {
        g.in_inv_scale[c] = net->in_inv_scale[c];
        g.lo[c] = net->box_lo[c];
        g.hi[c] = net->box_hi[c];
    }
    g.tol = tol;
    return g;
}
const MatConst& net_material(const mpm_net* net) { return net->mat; }
}  // namespace mpm

// closure.cu - the learned eddy-viscosity closure: training data from
// box-filtered, 2x-restricted snapshots of a fine run of this solver, and
// the MLP's forward, backward and Adam kernels (no counterpart in the
// reference, whose collision uses a constant tau per phase, lbm.cu:158-170).
//
// Network (same as the collide kernel's mlp_nu_t): features x = (Pi_xx,
// Pi_yy, Pi_zz, Pi_xy, Pi_xz, Pi_yz, phi, |grad phi|), x' = (x - mean) *
// inv_scale, h1 = SiLU(W1 x' + b1), h2 = SiLU(W2 h1 + b2),
// nu_t = out_scale * softplus(w3 . h2 + b3). Training loss per sample:
// (softplus(z) - target / out_scale)^2, averaged over a minibatch.
//
// Training data. A coarse node X of the 2x-coarser grid sits on fine node
// 2X. Fine rho, u, phi and the products u_a u_b are averaged over the 3x3x3
// fine box around 2X (box filter + restriction). On the coarse grid:
//   S_ab   = (d_a u_b + d_b u_a) / 2, central differences (coarse spacing 1),
//   tau_ab = <u_a u_b> - <u_a><u_b> (sub-filter stress),
//   target nu_t = min(kMaxNuT, max(0, -dev(tau) : S / (2 S : S))), 0 where
//            S : S < kMinStrain2 (least-squares eddy viscosity, coarse
//            lattice units),
//   features: Pi = -2 rho cs^2 tau0 dev(S) (the non-equilibrium stress the
//            coarse solver carries, Chapman-Enskog, tau0 its molecular
//            relaxation time), phi, |grad phi| (D3Q19 lattice gradient, as
//            the solver's normals stencil).
//
// Interface width. The same sample nodes give the thickness of the phase
// interface: for a tanh profile, sum phi (1 - phi) / sum |grad phi| is a
// quarter of the width W. Measured on the filtered coarse field (coarse
// units) and on the fine field at the sample's fine node 2X (fine units, the
// solver's own |grad phi|), their ratio is the factor by which the coarse
// run's interface sharpening gamma must grow for its equilibrium interface
// (W proportional to 1 / gamma at the fixed phase mobility) to have the
// filtered fine width; the coarse grid otherwise resolves an interface twice
// as thick in physical units.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "../../include/pflbm.h"
#include "engine.h"
#include "faults.h"
#include "gridbar.cuh"
#include "kernels.cuh"
#include "packed.cuh"
#include "widen.cuh"

namespace {

using pflbm::kMlpBlob;
using pflbm::kMlpH;
using pflbm::kMlpIn;
using pflbm::kMlpParams;

static_assert(kMlpParams == PFLBM_MLP_PARAMS && kMlpBlob == PFLBM_MLP_BLOB, "closure blob layout");
static_assert(kMlpParams == pflbm::kMlpParamFloats && kMlpBlob == pflbm::kMlpBlobFloats, "closure blob layout");
static_assert(pflbm::kMlpStrength == kMlpBlob - 1, "strength is the last blob entry");

constexpr int kSB = 128;            // samples per training block
constexpr int kCoarseFields = 11;   // rho, ux, uy, uz, phi, tau_xx, tau_yy, tau_zz, tau_xy, tau_xz, tau_yz
constexpr int kLossBlocks = 1024;
constexpr float kMinStrain2 = 1e-10f;  // S:S below which the target is 0
constexpr float kMaxNuT = 2e-3f;       // cap of the target eddy viscosity (lattice units)

int fail(int code, const std::string &msg) {
    pflbm::set_error(msg);
    return code;
}

int cuda_fail(cudaError_t e, const char *what) {
    cudaGetLastError();
    return fail(PFLBM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

__host__ __device__ inline uint64_t mix64(uint64_t x) {
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

// (the correctly rounded reciprocal is the correctly rounded quotient 1 / x,
// in fewer instructions than a division)
__device__ __forceinline__ float sigmoidf_(float a) { return __frcp_rn(1.0f + expf(-a)); }

// ------------------------------------------------------------- data
// Box filter and restriction in FP64, bound by the FP64 unit. A thread owns a
// coarse column (i, j) of a z chunk, sums every fine plane of its boxes once
// and carries plane 2k+1 on to the next coarse plane; the floats are widened on
// the integer units: 251 FP64 instructions per coarse node by count (275
// executed, the chunks' first planes included) instead of 455 with the
// conversions, 64x64x256 coarse nodes 910 -> 560 us (753 with the conversions
// in FP64).
constexpr int kFilterX = 32, kFilterY = 4, kFilterPlanes = 8;
__global__ void __launch_bounds__(kFilterX *kFilterY) k_filter_restrict(const float *__restrict__ macro, uint64_t Nf,
                                                                        int nxf, int nyf, int nzf, int nxc, int nyc,
                                                                        int nzc, float *__restrict__ coarse) {
    const uint64_t Nc = uint64_t(nxc) * nyc * nzc;
    const int i = int(blockIdx.x) * kFilterX + threadIdx.x, j = int(blockIdx.y) * kFilterY + threadIdx.y;
    if (i >= nxc || j >= nyc) return;
    const int xm = max(2 * i - 1, 0), x0 = min(2 * i, nxf - 1), xp = min(2 * i + 1, nxf - 1);
    const int slot[5] = {pflbm::M_RHO, pflbm::M_UX, pflbm::M_UY, pflbm::M_UZ, pflbm::M_PHI};
    // sums over the x triple of fine row y, plane z
    auto row = [&](int y, int z, double (&r)[kCoarseFields]) {
        const uint64_t base = uint64_t(nxf) * (uint64_t(min(max(y, 0), nyf - 1)) + uint64_t(nyf) * z);
        float q[15];
        double v[15];
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const float *p = macro + slot[f] * Nf + base;
            q[3 * f] = p[xm], q[3 * f + 1] = p[x0], q[3 * f + 2] = p[xp];
        }
        pflbm::widen_all(q, v);
#pragma unroll
        for (int f = 0; f < 5; ++f) r[f] = v[3 * f] + v[3 * f + 1] + v[3 * f + 2];
        constexpr int A[6] = {1, 2, 3, 1, 1, 2}, B[6] = {1, 2, 3, 2, 3, 3};
#pragma unroll
        for (int k = 0; k < 6; ++k)
            r[5 + k] = fma(v[3 * A[k] + 2], v[3 * B[k] + 2],
                           fma(v[3 * A[k] + 1], v[3 * B[k] + 1], v[3 * A[k]] * v[3 * B[k]]));
    };
    // sums over the three rows of the box in fine plane z (clamped)
    auto plane = [&](int z, double (&s)[kCoarseFields]) {
        z = min(max(z, 0), nzf - 1);
        double r[kCoarseFields];
        row(2 * j, z, s);
#pragma unroll
        for (int dy = -1; dy <= 1; dy += 2) {
            row(2 * j + dy, z, r);
#pragma unroll
            for (int f = 0; f < kCoarseFields; ++f) s[f] += r[f];
        }
    };
    const int k0 = int(blockIdx.z) * kFilterPlanes, k1 = min(k0 + kFilterPlanes, nzc);
    double below[kCoarseFields], s[kCoarseFields], above[kCoarseFields];
    plane(2 * k0 - 1, below);
    for (int k = k0; k < k1; ++k) {
        plane(2 * k, s);
        plane(2 * k + 1, above);
        double m[kCoarseFields];
#pragma unroll
        for (int f = 0; f < kCoarseFields; ++f) {
            m[f] = (below[f] + s[f] + above[f]) * (1.0 / 27.0);
            below[f] = above[f];
        }
        const uint64_t c = uint64_t(i) + uint64_t(nxc) * (uint64_t(j) + uint64_t(nyc) * k);
#pragma unroll
        for (int f = 0; f < 5; ++f) coarse[f * Nc + c] = float(m[f]);
        coarse[5 * Nc + c] = float(m[5] - m[1] * m[1]);
        coarse[6 * Nc + c] = float(m[6] - m[2] * m[2]);
        coarse[7 * Nc + c] = float(m[7] - m[3] * m[3]);
        coarse[8 * Nc + c] = float(m[8] - m[1] * m[2]);
        coarse[9 * Nc + c] = float(m[9] - m[1] * m[3]);
        coarse[10 * Nc + c] = float(m[10] - m[2] * m[3]);
    }
}

// Samples at coarse nodes 2 <= i,j,k <= n-3 with i % stride == 0 and
// j % stride == 0, written in (k, j, i) order from `base`.
// Each block also writes its sums of phi(1-phi) and |grad phi| on the
// filtered coarse field and on the fine field at 2X (width[blockIdx.x * 4 +
// 0..3], FP64, summed in block order on the host).
constexpr int kMakeThreads = 256, kMakeBlocks = 1216;
__global__ void __launch_bounds__(kMakeThreads) k_make_samples(const float *__restrict__ coarse, int nxc, int nyc,
                                                               int nzc, int stride, float tau_w, float tau_o, int i0,
                                                               int ni, int j0, int nj, float *__restrict__ X,
                                                               float *__restrict__ Y, uint64_t base,
                                                               const float *__restrict__ macro, uint64_t Nf, int nxf,
                                                               int nyf, double *__restrict__ width) {
    const uint64_t Nc = uint64_t(nxc) * nyc * nzc;
    const uint64_t total = uint64_t(ni) * nj * (nzc - 4);
    double wsum[4] = {0.0, 0.0, 0.0, 0.0};
    for (uint64_t s = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; s < total; s += uint64_t(gridDim.x) * blockDim.x) {
        const int ii = int(s % ni), jj = int((s / ni) % nj), kk = int(s / (uint64_t(ni) * nj));
        const int i = i0 + ii * stride, j = j0 + jj * stride, k = 2 + kk;
        auto at = [&](int f, int x, int y, int z) -> float {
            return coarse[f * Nc + uint64_t(x) + uint64_t(nxc) * (uint64_t(y) + uint64_t(nyc) * z)];
        };
        float g[3][3];  // g[a][b] = d_a u_b
        for (int b = 0; b < 3; ++b) {
            g[0][b] = 0.5f * (at(1 + b, i + 1, j, k) - at(1 + b, i - 1, j, k));
            g[1][b] = 0.5f * (at(1 + b, i, j + 1, k) - at(1 + b, i, j - 1, k));
            g[2][b] = 0.5f * (at(1 + b, i, j, k + 1) - at(1 + b, i, j, k - 1));
        }
        const float sxx = g[0][0], syy = g[1][1], szz = g[2][2];
        const float sxy = 0.5f * (g[0][1] + g[1][0]), sxz = 0.5f * (g[0][2] + g[2][0]), syz = 0.5f * (g[1][2] + g[2][1]);
        const float tr = (sxx + syy + szz) / 3.0f;
        const float dxx = sxx - tr, dyy = syy - tr, dzz = szz - tr;
        const float rho = at(0, i, j, k), phi = at(4, i, j, k);
        const float tau0 = (1.0f - phi) * tau_w + phi * tau_o;
        const float c = -2.0f * rho * tau0 / 3.0f;
        // |grad phi| with the D3Q19 lattice gradient (3 sum_q w_q c_q phi(x + c_q))
        float gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
        for (int q = 1; q < 19; ++q) {
            const float w = pflbm::weight<19>(q) * at(4, i + pflbm::kCX[q], j + pflbm::kCY[q], k + pflbm::kCZ[q]);
            gx += w * pflbm::kCX[q];
            gy += w * pflbm::kCY[q];
            gz += w * pflbm::kCZ[q];
        }
        const float ind = 3.0f * sqrtf(gx * gx + gy * gy + gz * gz);
        // least-squares eddy viscosity of the sub-filter stress
        const float txx = at(5, i, j, k), tyy = at(6, i, j, k), tzz = at(7, i, j, k);
        const float txy = at(8, i, j, k), txz = at(9, i, j, k), tyz = at(10, i, j, k);
        const float ttr = (txx + tyy + tzz) / 3.0f;
        const float num = -((txx - ttr) * sxx + (tyy - ttr) * syy + (tzz - ttr) * szz +
                            2.0f * (txy * sxy + txz * sxz + tyz * syz));
        const float den = 2.0f * (sxx * sxx + syy * syy + szz * szz + 2.0f * (sxy * sxy + sxz * sxz + syz * syz));
        // quiescent nodes (S:S below kMinStrain2) carry no information on
        // nu_t; the cap removes the heavy tail of near-zero strain rates
        const float nu = den > 2.0f * kMinStrain2 ? fminf(fmaxf(0.0f, num / den), kMaxNuT) : 0.0f;
        float *x = X + (base + s) * kMlpIn;
        x[0] = c * dxx; x[1] = c * dyy; x[2] = c * dzz;
        x[3] = c * sxy; x[4] = c * sxz; x[5] = c * syz;
        x[6] = phi; x[7] = ind;
        Y[base + s] = nu;
        const uint64_t f = uint64_t(2 * i) + uint64_t(nxf) * (uint64_t(2 * j) + uint64_t(nyf) * uint64_t(2 * k));
        const double phf = macro[pflbm::M_PHI * Nf + f], indf = macro[pflbm::M_IND * Nf + f];
        wsum[0] += double(phi) * (1.0 - double(phi));
        wsum[1] += double(ind);
        wsum[2] += phf * (1.0 - phf);
        wsum[3] += indf;
    }
    __shared__ double red[4][kMakeThreads];
    for (int q = 0; q < 4; ++q) red[q][threadIdx.x] = wsum[q];
    __syncthreads();
    for (int h = kMakeThreads / 2; h > 0; h >>= 1) {
        if (int(threadIdx.x) < h)
            for (int q = 0; q < 4; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x < 4) width[blockIdx.x * 4 + threadIdx.x] = red[threadIdx.x][0];
}

// FP64 sums of x_k, x_k^2 (k < 8), y, y^2 per block.
__global__ void __launch_bounds__(256) k_stats(const float *__restrict__ X, const float *__restrict__ Y, uint64_t n,
                                               double *__restrict__ partial) {
    double acc[18] = {0};
    for (uint64_t s = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; s < n; s += uint64_t(gridDim.x) * blockDim.x) {
        for (int k = 0; k < kMlpIn; ++k) {
            const double v = X[s * kMlpIn + k];
            acc[k] += v;
            acc[8 + k] += v * v;
        }
        const double y = Y[s];
        acc[16] += y;
        acc[17] += y * y;
    }
    __shared__ double sh[18][256];
    for (int f = 0; f < 18; ++f) sh[f][threadIdx.x] = acc[f];
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st)
            for (int f = 0; f < 18; ++f) sh[f][threadIdx.x] += sh[f][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x < 18) partial[blockIdx.x * 18 + threadIdx.x] = sh[threadIdx.x][0];
}

// ------------------------------------------------------------- network
struct Act {
    float xn[kSB][kMlpIn];
    float h1[kSB][kMlpH + 1];   // +1: bank-conflict padding
    float da1[kSB][kMlpH + 1];
    float h2[kSB][kMlpH + 1];
    float da2[kSB][kMlpH + 1];
    float dz[kSB];
    float loss[kSB];
};

// Forward + backward over one block of kSB samples. Sample index: k for
// mode 0 (the first n samples in order), else a hash of (seed, iteration, k)
// modulo n. Per-block gradient sums -> gpart[block][0..kMlpParams), the
// block's loss sum -> gpart[block][kMlpParams].
__global__ void __launch_bounds__(kSB) k_mlp_grad(const float *__restrict__ blob, const float *__restrict__ X,
                                                  const float *__restrict__ Y, uint64_t n, int mode, uint64_t seed,
                                                  uint64_t iter, uint64_t count, float *__restrict__ gpart) {
    __shared__ float w[kMlpBlob];
    extern __shared__ unsigned char dyn[];
    Act &A = *reinterpret_cast<Act *>(dyn);
    for (int i = threadIdx.x; i < kMlpBlob; i += kSB) w[i] = blob[i];
    __syncthreads();
    const int t = threadIdx.x;
    const uint64_t k = blockIdx.x * uint64_t(kSB) + t;
    const bool valid = k < count;
    uint64_t idx = 0;
    if (valid) idx = mode == 0 ? k : mix64(seed * 0x9E3779B97F4A7C15ull + mix64(iter * 0x100000001B3ull + k)) % n;
    const float out_scale = w[pflbm::kMlpOutScale];
    float a1[kMlpH], a2[kMlpH];
    float xn[kMlpIn];
    for (int q = 0; q < kMlpIn; ++q)
        xn[q] = valid ? (X[idx * kMlpIn + q] - w[pflbm::kMlpMean + q]) * w[pflbm::kMlpInvScale + q] : 0.0f;
#pragma unroll
    for (int i = 0; i < kMlpH; ++i) {
        float s = w[pflbm::kMlpB1 + i];
#pragma unroll
        for (int q = 0; q < kMlpIn; ++q) s += w[pflbm::kMlpW1 + i * kMlpIn + q] * xn[q];
        a1[i] = s;
        A.h1[t][i] = s * sigmoidf_(s);
    }
    float z = w[pflbm::kMlpB3];
#pragma unroll 4
    for (int j = 0; j < kMlpH; ++j) {
        float s = w[pflbm::kMlpB2 + j];
#pragma unroll
        for (int i = 0; i < kMlpH; ++i) s += w[pflbm::kMlpW2 + j * kMlpH + i] * A.h1[t][i];
        a2[j] = s;
        const float h = s * sigmoidf_(s);
        A.h2[t][j] = h;
        z += w[pflbm::kMlpW3 + j] * h;
    }
    const float sp = fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z)));
    const float r = valid ? sp - Y[idx] / out_scale : 0.0f;
    const float dz = 2.0f * r * sigmoidf_(z);
    A.dz[t] = valid ? dz : 0.0f;
    A.loss[t] = r * r;
#pragma unroll
    for (int q = 0; q < kMlpIn; ++q) A.xn[t][q] = xn[q];
#pragma unroll
    for (int j = 0; j < kMlpH; ++j) {
        const float sg = sigmoidf_(a2[j]);
        A.da2[t][j] = valid ? dz * w[pflbm::kMlpW3 + j] * sg * (1.0f + a2[j] * (1.0f - sg)) : 0.0f;
    }
#pragma unroll 4
    for (int i = 0; i < kMlpH; ++i) {
        float dh = 0.0f;
#pragma unroll
        for (int j = 0; j < kMlpH; ++j) dh += w[pflbm::kMlpW2 + j * kMlpH + i] * A.da2[t][j];
        const float sg = sigmoidf_(a1[i]);
        A.da1[t][i] = dh * sg * (1.0f + a1[i] * (1.0f - sg));
    }
    __syncthreads();
    // parameter gradients: sums over the block's samples, in sample order
    float *g = gpart + size_t(blockIdx.x) * (kMlpParams + 1);
    for (int p = t; p <= kMlpParams; p += kSB) {
        float acc = 0.0f;
        if (p < pflbm::kMlpB1) {  // W1[i][q]
            const int i = p / kMlpIn, q = p % kMlpIn;
            for (int s = 0; s < kSB; ++s) acc += A.da1[s][i] * A.xn[s][q];
        } else if (p < pflbm::kMlpW2) {  // b1[i]
            const int i = p - pflbm::kMlpB1;
            for (int s = 0; s < kSB; ++s) acc += A.da1[s][i];
        } else if (p < pflbm::kMlpB2) {  // W2[j][i]
            const int j = (p - pflbm::kMlpW2) / kMlpH, i = (p - pflbm::kMlpW2) % kMlpH;
            for (int s = 0; s < kSB; ++s) acc += A.da2[s][j] * A.h1[s][i];
        } else if (p < pflbm::kMlpW3) {  // b2[j]
            const int j = p - pflbm::kMlpB2;
            for (int s = 0; s < kSB; ++s) acc += A.da2[s][j];
        } else if (p < pflbm::kMlpB3) {  // w3[j]
            const int j = p - pflbm::kMlpW3;
            for (int s = 0; s < kSB; ++s) acc += A.dz[s] * A.h2[s][j];
        } else if (p == pflbm::kMlpB3) {
            for (int s = 0; s < kSB; ++s) acc += A.dz[s];
        } else {  // loss sum
            for (int s = 0; s < kSB; ++s)
                if (blockIdx.x * uint64_t(kSB) + s < count) acc += A.loss[s];
        }
        g[p] = acc;
    }
}

// ------------------------------------------- network on the tensor cores
// The same forward + backward over blocks of kSB = 128 samples with every
// matrix product on the tensor cores: warp-level mma.m16n8k8 with TF32
// operands (10-bit mantissa, operands rounded to nearest) and FP32
// accumulation. A pair of warps owns 32 samples, each warp one 16-row tile
// of them up to the weight gradients, whose output rows they then share:
//   layer 1   A1 = Xn W1^T + b1       (16 x 8 x 8 per column block)
//   layer 2   A2 = H1 W2^T + b2       (K = 32: four k steps)
//   backward  dH1 = dA2 W2            (K = 32)
//   weights   dW2 = dA2^T H1, dW1 = dA1^T Xn   (K = the pair's 32 samples)
// and the elementwise parts (SiLU, softplus, bias and w3 sums) in FP32. The
// four pairs' partial gradients are summed in pair order in FP32 (the block's
// gradient, as k_mlp_grad's) and added to the CTA's FP64 sums.
//
// What bounds it is the dependent chain of one block (gather, two layers,
// two layers back, column sums), not the 112 MMAs per 32 samples. So the
// weights are laid out once as TF32 fragments in lane order (8-byte
// conflict-free loads instead of 4- and 8-way conflicts and a conversion per
// use), a sigmoid is evaluated once per unit instead of two or three times,
// and two warps share what one warp did: 2^20 samples 398 -> 226 us at 16
// warps per SM, 202 us at 24 (3790 warp instructions per 32 samples, 2.1 of 4
// issued per clock).
constexpr int kTcThreads = 2 * kSB;
constexpr int kTcPairs = kSB / 32;
constexpr int kTcX = 12;         // row stride of the Xn tile (words)
constexpr int kTcH = kMlpH + 4;  // row stride of the 32-wide tiles
// shared words: weight fragments and constants, then per pair Xn, H1 (TF32
// bits), dA2, dA1 (each first holding SiLU' of its units), dz, loss, the w3
// sums of the first tile; the pair's partial gradient takes the same place
// when the tiles have been read. With that, and W2's fragments read as scalars
// for the transposed product, three CTAs fit an SM (72 KB, 80 registers)
constexpr int kTcF1 = 0, kTcF2 = kTcF1 + 256, kTcB1 = kTcF2 + 1024, kTcB2 = kTcB1 + kMlpH,
              kTcW3 = kTcB2 + kMlpH, kTcMean = kTcW3 + kMlpH, kTcInv = kTcMean + kMlpIn, kTcB3 = kTcInv + kMlpIn,
              kTcScale = kTcB3 + 1, kTcWeights = kTcB3 + 4;
constexpr int kTcPairWords = 32 * kTcX + 3 * 32 * kTcH + 32 + 32 + 8 * 32;
constexpr int kTcPart = kMlpParams + 1;  // partial gradient + loss
constexpr int kTcAcc = (kTcPart + kTcThreads - 1) / kTcThreads;  // FP64 sums per thread
constexpr int kTcSmem = 4 * (kTcWeights + kTcPairs * kTcPairWords);
static_assert(kTcPart <= kTcPairWords, "the partial gradient takes the pair's tiles' place");
static_assert(kMlpH == 32 && kMlpIn == 8, "fragment layout");

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// D = A B + C, A 16x8 (row), B 8x8 (col), TF32 operands, FP32 accumulators.
__device__ __forceinline__ void mma_tf32_1688(float (&d)[4], const uint32_t (&a)[4], uint2 b) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

// The two warps of a pair (named barriers 1 .. kTcPairs; 0 is the block's).
__device__ __forceinline__ void pair_sync(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); }

// The blob as fragments: B operand words of lane (g = lane / 4, t = lane % 4)
// side by side, W1 and W2 by output column block and k step. Read past the L1, which another CTA's
// update of the blob does not invalidate.
__device__ __forceinline__ void tc_load_weights(float *s, const float *blob) {
    uint32_t *w = reinterpret_cast<uint32_t *>(s);
    constexpr int kPer = (kMlpBlob + kTcThreads - 1) / kTcThreads;
    float got[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (threadIdx.x + kTcThreads * k < kMlpBlob) got[k] = __ldcg(blob + threadIdx.x + kTcThreads * k);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int i = threadIdx.x + kTcThreads * k;
        const float v = got[k];
        if (i < pflbm::kMlpB1) {
            const int n = i >> 3, k = i & 7;
            w[kTcF1 + (((n >> 3) * 32 + (n & 7) * 4 + (k & 3)) * 2) + (k >> 2)] = to_tf32(v);
        } else if (i < pflbm::kMlpW2) {
            s[kTcB1 + i - pflbm::kMlpB1] = v;
        } else if (i < pflbm::kMlpB2) {
            const int j = (i - pflbm::kMlpW2) >> 5, c = (i - pflbm::kMlpW2) & 31;
            w[kTcF2 + (((j >> 3) * 4 + (c >> 3)) * 32 + (j & 7) * 4 + (c & 3)) * 2 + ((c >> 2) & 1)] = to_tf32(v);
        } else if (i < pflbm::kMlpW3) {
            s[kTcB2 + i - pflbm::kMlpB2] = v;
        } else if (i < pflbm::kMlpB3) {
            s[kTcW3 + i - pflbm::kMlpW3] = v;
        } else if (i == pflbm::kMlpB3) {
            s[kTcB3] = v;
        } else if (i < pflbm::kMlpInvScale) {
            s[kTcMean + i - pflbm::kMlpMean] = v;
        } else if (i < pflbm::kMlpOutScale) {
            s[kTcInv + i - pflbm::kMlpInvScale] = v;
        } else if (i == pflbm::kMlpOutScale) {
            s[kTcScale] = v;
        }
    }
}

// What a warp needs of its 16 samples of a block: lane l half a row (row
// l / 2) of features, lanes 0 .. 15 the target of row l.
struct TcRows {
    float4 x;
    float y;
    bool vx, vy;  // the rows exist (the last block is ragged)
};

__device__ __forceinline__ TcRows tc_fetch(const float *__restrict__ X, const float *__restrict__ Y, uint64_t n,
                                           int mode, uint64_t seed, uint64_t iter, uint64_t count, int block) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = uint64_t(block) * kSB + uint64_t(warp) * 16;
    TcRows r{make_float4(0.f, 0.f, 0.f, 0.f), 0.0f, base + (lane >> 1) < count, lane < 16 && base + lane < count};
    const uint64_t k = base + (lane >> 1);
    uint64_t idx = 0;
    if (r.vx) idx = mode == 0 ? k : mix64(seed * 0x9E3779B97F4A7C15ull + mix64(iter * 0x100000001B3ull + k)) % n;
    if (r.vx) r.x = __ldg(reinterpret_cast<const float4 *>(X + idx * kMlpIn) + (lane & 1));
    const uint64_t iy = __shfl_sync(0xffffffffu, idx, (2 * lane) & 31);
    if (r.vy) r.y = __ldg(Y + iy);
    return r;
}

// Gradient of one block's samples, added to the calling thread's FP64 sums
// (parameter threadIdx.x + kTcThreads j in acc[j]; the loss is the last one).
__device__ __forceinline__ void tc_block(float *s, const TcRows &rows, double (&acc)[kTcAcc]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pair = warp >> 1, half = warp & 1;  // this warp's rows: 16 half .. 16 half + 15 of the pair's 32
    const int g = lane >> 2, t = lane & 3;
    float *base = s + kTcWeights + pair * kTcPairWords;
    uint32_t *xs = reinterpret_cast<uint32_t *>(base);  // [32][kTcX], TF32
    uint32_t *h1s = xs + 32 * kTcX;                     // [32][kTcH], TF32
    float *da2s = base + 32 * kTcX + 32 * kTcH;         // [32][kTcH]
    float *da1s = da2s + 32 * kTcH;                     // [32][kTcH]
    float *dzs = da1s + 32 * kTcH;                      // [32]
    float *losses = dzs + 32;                           // [32]
    float *w3p = losses + 32;                           // [8][32]
    float *part = base;
    const uint2 *f1 = reinterpret_cast<const uint2 *>(s + kTcF1), *f2 = reinterpret_cast<const uint2 *>(s + kTcF2);
    // W2[8 kk + t (+4)][8 nt + g]: the word of lane (g, t) in the transposed product
    const uint32_t *f2t = reinterpret_cast<const uint32_t *>(s + kTcF2) + (t * 4 + (g & 3)) * 2 + (g >> 2);

    // normalised features
    {
        const int q = 4 * (lane & 1);
        const float *mean = s + kTcMean + q, *inv = s + kTcInv + q;
        const float4 x = rows.x;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (rows.vx)
            v = make_uint4(to_tf32((x.x - mean[0]) * inv[0]), to_tf32((x.y - mean[1]) * inv[1]),
                           to_tf32((x.z - mean[2]) * inv[2]), to_tf32((x.w - mean[3]) * inv[3]));
        *reinterpret_cast<uint4 *>(&xs[(16 * half + (lane >> 1)) * kTcX + q]) = v;
    }
    const float target = rows.vy ? rows.y / s[kTcScale] : 0.0f;
    __syncwarp();

    const int r0 = 16 * half + g;  // fragment rows r0 and r0 + 8, columns 8 nt + 2 t (+1)
    // layer 1: a1 = Xn W1^T + b1; h1 = SiLU(a1) and SiLU'(a1) to shared memory
    {
        const uint32_t a[4] = {xs[r0 * kTcX + t], xs[(r0 + 8) * kTcX + t], xs[r0 * kTcX + t + 4],
                               xs[(r0 + 8) * kTcX + t + 4]};
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const float c0 = s[kTcB1 + 8 * nt + 2 * t], c1 = s[kTcB1 + 8 * nt + 2 * t + 1];
            float d[4] = {c0, c1, c0, c1};
            mma_tf32_1688(d, a, f1[nt * 32 + lane]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float sg = sigmoidf_(d[e]);
                const int at = (r0 + (e >= 2 ? 8 : 0)) * kTcH + 8 * nt + 2 * t + (e & 1);
                h1s[at] = to_tf32(d[e] * sg);
                da1s[at] = sg * (1.0f + d[e] * (1.0f - sg));
            }
        }
    }
    __syncwarp();
    // layer 2: a2 = H1 W2^T + b2; z = w3 . SiLU(a2) + b3 per sample
    float h2[4][4], zp[2] = {0.f, 0.f};
    {
        uint32_t a[4][4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            a[kk][0] = h1s[r0 * kTcH + 8 * kk + t];
            a[kk][1] = h1s[(r0 + 8) * kTcH + 8 * kk + t];
            a[kk][2] = h1s[r0 * kTcH + 8 * kk + t + 4];
            a[kk][3] = h1s[(r0 + 8) * kTcH + 8 * kk + t + 4];
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const float c0 = s[kTcB2 + 8 * nt + 2 * t], c1 = s[kTcB2 + 8 * nt + 2 * t + 1];
            float d[4] = {c0, c1, c0, c1};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) mma_tf32_1688(d, a[kk], f2[(nt * 4 + kk) * 32 + lane]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float sg = sigmoidf_(d[e]);
                h2[nt][e] = d[e] * sg;
                da2s[(r0 + (e >= 2 ? 8 : 0)) * kTcH + 8 * nt + 2 * t + (e & 1)] = sg * (1.0f + d[e] * (1.0f - sg));
                zp[e >> 1] = __fmaf_rn(s[kTcW3 + 8 * nt + 2 * t + (e & 1)], h2[nt][e], zp[e >> 1]);
            }
        }
    }
    // complete z over the 4 lanes of a group, then dz per row to shared memory
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        zp[h] += __shfl_xor_sync(0xffffffffu, zp[h], 1);
        zp[h] += __shfl_xor_sync(0xffffffffu, zp[h], 2);
    }
    if (t == 0) {
        dzs[r0] = zp[0] + s[kTcB3];
        dzs[r0 + 8] = zp[1] + s[kTcB3];
    }
    __syncwarp();
    if (lane < 16) {
        const float z = dzs[16 * half + lane];
        const float sp = fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z)));
        const float r = rows.vy ? sp - target : 0.0f;
        losses[16 * half + lane] = rows.vy ? r * r : 0.0f;
        dzs[16 * half + lane] = rows.vy ? 2.0f * r * sigmoidf_(z) : 0.0f;
    }
    __syncwarp();
    // backward: dA2 = dz w3 SiLU'(a2); the w3 sums of the pair run over the
    // first warp's rows, then over the second's
    const float dz0 = dzs[r0], dz1 = dzs[r0 + 8];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = 8 * nt + 2 * t + (e & 1), at = (r0 + (e >= 2 ? 8 : 0)) * kTcH + col;
            da2s[at] = (e >= 2 ? dz1 : dz0) * s[kTcW3 + col] * da2s[at];
        }
    if (half == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            w3p[k * 32 + lane] = __fmaf_rn(dz1, h2[k >> 1][2 + (k & 1)], __fmul_rn(dz0, h2[k >> 1][k & 1]));
    }
    __syncwarp();
    // dH1 = dA2 W2, dA1 = dH1 SiLU'(a1)
    {
        uint32_t a[4][4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            a[kk][0] = to_tf32(da2s[r0 * kTcH + 8 * kk + t]);
            a[kk][1] = to_tf32(da2s[(r0 + 8) * kTcH + 8 * kk + t]);
            a[kk][2] = to_tf32(da2s[r0 * kTcH + 8 * kk + t + 4]);
            a[kk][3] = to_tf32(da2s[(r0 + 8) * kTcH + 8 * kk + t + 4]);
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                mma_tf32_1688(d, a[kk], make_uint2(f2t[(kk * 4 + nt) * 64], f2t[(kk * 4 + nt) * 64 + 32]));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int at = (r0 + (e >= 2 ? 8 : 0)) * kTcH + 8 * nt + 2 * t + (e & 1);
                da1s[at] = d[e] * da1s[at];
            }
        }
    }
    pair_sync(pair);
    // weight gradients over the pair's 32 samples (K): this warp the output
    // rows 16 half .. 16 half + 15
    float dw2[4][4], dw1[4] = {0.f, 0.f, 0.f, 0.f};
    {
        uint32_t a[4][4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            a[kk][0] = to_tf32(da2s[(8 * kk + t) * kTcH + r0]);
            a[kk][1] = to_tf32(da2s[(8 * kk + t) * kTcH + r0 + 8]);
            a[kk][2] = to_tf32(da2s[(8 * kk + t + 4) * kTcH + r0]);
            a[kk][3] = to_tf32(da2s[(8 * kk + t + 4) * kTcH + r0 + 8]);
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {  // dW2[j][i] = sum_s dA2[s][j] H1[s][i]
#pragma unroll
            for (int e = 0; e < 4; ++e) dw2[nt][e] = 0.f;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                mma_tf32_1688(dw2[nt], a[kk], make_uint2(h1s[(8 * kk + t) * kTcH + 8 * nt + g],
                                                         h1s[(8 * kk + t + 4) * kTcH + 8 * nt + g]));
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {  // dW1[i][q] = sum_s dA1[s][i] Xn[s][q]
            const uint32_t b[4] = {to_tf32(da1s[(8 * kk + t) * kTcH + r0]), to_tf32(da1s[(8 * kk + t) * kTcH + r0 + 8]),
                                   to_tf32(da1s[(8 * kk + t + 4) * kTcH + r0]),
                                   to_tf32(da1s[(8 * kk + t + 4) * kTcH + r0 + 8])};
            mma_tf32_1688(dw1, b, make_uint2(xs[(8 * kk + t) * kTcX + g], xs[(8 * kk + t + 4) * kTcX + g]));
        }
    }
    // bias gradients: column sums over the pair's samples, b1 by the first
    // warp, b2 by the second; b3 and the loss by the first, w3 by the second
    float sb = 0.f, sdz = 0.f, sl = 0.f, dw3[8];
    {
        const float *col = (half == 0 ? da1s : da2s) + lane;
#pragma unroll
        for (int r = 0; r < 32; ++r) sb += col[r * kTcH];
    }
    if (half == 0) {
        sdz = dzs[lane], sl = losses[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sdz += __shfl_xor_sync(0xffffffffu, sdz, o);
            sl += __shfl_xor_sync(0xffffffffu, sl, o);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float v = __fmaf_rn(dz0, h2[k >> 1][k & 1], w3p[k * 32 + lane]);
            v = __fmaf_rn(dz1, h2[k >> 1][2 + (k & 1)], v);
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            dw3[k] = v;
        }
    }
    pair_sync(pair);  // the tiles have been read
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            part[pflbm::kMlpW2 + (r0 + (e >= 2 ? 8 : 0)) * kMlpH + 8 * nt + 2 * t + (e & 1)] = dw2[nt][e];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        part[pflbm::kMlpW1 + (r0 + (e >= 2 ? 8 : 0)) * kMlpIn + 2 * t + (e & 1)] = dw1[e];
    part[(half == 0 ? pflbm::kMlpB1 : pflbm::kMlpB2) + lane] = sb;
    if (half == 0 && lane == 0) {
        part[pflbm::kMlpB3] = sdz;
        part[kMlpParams] = sl;
    }
    if (half == 1 && g == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) part[pflbm::kMlpW3 + 8 * (k >> 1) + 2 * t + (k & 1)] = dw3[k];
    }
    __syncthreads();
    // the block's sums, pairs in order
    const float *parts = s + kTcWeights;
#pragma unroll
    for (int j = 0; j < kTcAcc; ++j) {
        const int p = threadIdx.x + kTcThreads * j;
        if (p <= kMlpParams) {
            float v = 0.0f;
#pragma unroll
            for (int q = 0; q < kTcPairs; ++q) v += parts[q * kTcPairWords + p];
            acc[j] += v;
        }
    }
    __syncthreads();
}

// One parameter's sum over the CTAs' rows of gsum[cta][kTcPart], for the
// kSumP parameters from p0 on: 16 groups of threads take every 16th row each,
// then the groups are added in order. Every parameter's rows are in flight at
// once; one thread per parameter and row after row took 20 us for 128 rows
// and 1.16 ms for 8192. The sum is the return value of the threads of group 0
// (tid < kSumP; parameter p0 + tid).
constexpr int kSumP = 16, kSumG = kTcThreads / kSumP;
constexpr int kSumCtas = (kTcPart + kSumP - 1) / kSumP;  // CTAs that cover all parameters

__device__ __forceinline__ double tc_sum_rows(const double *gsum, int rows, int p0, double *red) {
    const int p = p0 + int(threadIdx.x) % kSumP, grp = int(threadIdx.x) / kSumP;
    double v = 0.0;
    if (p <= kMlpParams) {
#pragma unroll 8
        for (int r = grp; r < rows; r += kSumG) v += __ldcg(gsum + size_t(r) * kTcPart + p);
    }
    red[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < kSumP) {
        double q[4];  // four short chains: an FP64 addition takes about 60 cycles here
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = red[k * kSumP + threadIdx.x];
#pragma unroll
        for (int k = 4; k < kSumG; ++k) q[k & 3] += red[k * kSumP + threadIdx.x];
        v = (q[0] + q[1]) + (q[2] + q[3]);
    }
    return v;
}

// Gradient of the first `count` samples: every CTA runs its share of the
// blocks and writes its FP64 sums as a row of gsum; k_grad_rows adds the rows.
__global__ void __launch_bounds__(kTcThreads, 3) k_mlp_grad_tc(const float *__restrict__ blob,
                                                               const float *__restrict__ X,
                                                               const float *__restrict__ Y, uint64_t n,
                                                               uint64_t count, int blocks, double *__restrict__ gsum) {
    extern __shared__ __align__(16) float tcs[];
    tc_load_weights(tcs, blob);
    double acc[kTcAcc] = {};
    TcRows rows = tc_fetch(X, Y, n, 0, 0, 0, count, blockIdx.x);
    __syncthreads();
    for (int b = blockIdx.x; b < blocks; b += gridDim.x) {
        const TcRows now = rows;
        // the next block's samples arrive while this one is computed
        if (b + int(gridDim.x) < blocks) rows = tc_fetch(X, Y, n, 0, 0, 0, count, b + gridDim.x);
        tc_block(tcs, now, acc);
    }
#pragma unroll
    for (int j = 0; j < kTcAcc; ++j) {
        const int p = threadIdx.x + kTcThreads * j;
        if (p <= kMlpParams) gsum[size_t(blockIdx.x) * kTcPart + p] = acc[j];
    }
}

__global__ void __launch_bounds__(kTcThreads) k_grad_rows(const double *gsum, int rows, double *__restrict__ grad) {
    __shared__ double red[kTcThreads];
    const double v = tc_sum_rows(gsum, rows, blockIdx.x * kSumP, red);
    const int p = blockIdx.x * kSumP + threadIdx.x;
    if (threadIdx.x < kSumP && p <= kMlpParams) grad[p] = v;
}

// Adam on one parameter, rounded op by op (no contraction left to the
// compiler), so that every kernel that calls it moves a parameter alike.
__device__ __forceinline__ void adam_update(float g, float lr, float beta1, float beta2, float eps, float c1, float c2,
                                            float &m, float &v, float &w) {
    m = __fmaf_rn(1.0f - beta1, g, __fmul_rn(beta1, m));
    v = __fmaf_rn(__fmul_rn(1.0f - beta2, g), g, __fmul_rn(beta2, v));
    w = __fsub_rn(w, __fdiv_rn(__fmul_rn(lr, __fdiv_rn(m, c1)), __fadd_rn(__fsqrt_rn(__fdiv_rn(v, c2)), eps)));
}

// A stretch of training iterations in ONE cooperative launch. An iteration is
// short (a few us) and strictly serial, so launches and a sum over the blocks
// by a few threads were most of it. Here every CTA keeps its place: gradient
// of its blocks into its row of gsum, grid barrier, Adam on the 16 parameters
// that the CTA owns, grid barrier, the new blob as
// fragments. The next iteration's samples do not depend on the parameters and
// are fetched while the CTA waits at the first barrier. 16 384 samples per iteration: 36 us
// (two launches) -> 11.7 us, about half of it the block, the rest its FP64 row,
// the sums, the barriers and the weights.
constexpr int kTrainChunk = 128;  // iterations per launch
struct TrainArgs {
    float *blob, *m, *v;
    const float *X, *Y;
    uint64_t n, seed, iter0, count;
    int blocks, iterations, log0;
    float inv_count, lr, beta1, beta2, eps;
    double *gsum, *loss_log;
    unsigned int *arrived;  // the launch's grid barriers, 0 before it
    unsigned int *err;
    float c1[kTrainChunk], c2[kTrainChunk];  // 1 - beta^t of the bias corrections
};

__global__ void __launch_bounds__(kTcThreads, 2) k_mlp_train(const __grid_constant__ TrainArgs a) {
    extern __shared__ __align__(16) float tcs[];
    __shared__ double red[kTcThreads];
    __shared__ int s_ok;
    // behind a launch whose barrier ran out nothing moves any more
    if (__syncthreads_or(__ldcg(a.err) != 0u)) return;
    const int rows_used = min(int(gridDim.x), a.blocks);  // the CTAs that have a block
    const bool has = int(blockIdx.x) < a.blocks;
    TcRows rows{};
    if (has) rows = tc_fetch(a.X, a.Y, a.n, 1, a.seed, a.iter0, a.count, blockIdx.x);
    for (int it = 0; it < a.iterations; ++it) {
        tc_load_weights(tcs, a.blob);
        __syncthreads();
        if (has) {
            double acc[kTcAcc] = {};
            for (int b = blockIdx.x; b < a.blocks; b += gridDim.x) {
                const TcRows now = rows;
                if (b + int(gridDim.x) < a.blocks)
                    rows = tc_fetch(a.X, a.Y, a.n, 1, a.seed, a.iter0 + it, a.count, b + gridDim.x);
                tc_block(tcs, now, acc);
            }
#pragma unroll
            for (int j = 0; j < kTcAcc; ++j) {
                const int k = threadIdx.x + kTcThreads * j;
                if (k <= kMlpParams) __stcg(a.gsum + size_t(blockIdx.x) * kTcPart + k, acc[j]);
            }
        }
        pflbm::grid_arrive(a.arrived);
        if (has && it + 1 < a.iterations) rows = tc_fetch(a.X, a.Y, a.n, 1, a.seed, a.iter0 + it + 1, a.count, blockIdx.x);
        if (!pflbm::grid_wait(a.arrived, gridDim.x, 2 * it, a.err, &s_ok)) return;
        // 16 parameters per CTA (more where fewer CTAs than that are resident)
        for (int c = blockIdx.x; c < kSumCtas; c += gridDim.x) {
            const int p = c * kSumP + threadIdx.x;
            const bool owner = threadIdx.x < kSumP && p < kMlpParams;
            float m = 0.0f, v = 0.0f, w = 0.0f;
            if (owner) m = a.m[p], v = a.v[p], w = __ldcg(a.blob + p);
            const double s = tc_sum_rows(a.gsum, rows_used, c * kSumP, red);
            if (owner) {
                const float g = float(s) * a.inv_count;
                adam_update(g, a.lr, a.beta1, a.beta2, a.eps, a.c1[it], a.c2[it], m, v, w);
                a.m[p] = m;
                a.v[p] = v;
                __stcg(a.blob + p, w);
            } else if (threadIdx.x < kSumP && p == kMlpParams) {
                a.loss_log[a.log0 + it] = s * a.inv_count;
            }
            if (c + int(gridDim.x) < kSumCtas) __syncthreads();  // red is written again
        }
        pflbm::grid_arrive(a.arrived);
        if (!pflbm::grid_wait(a.arrived, gridDim.x, 2 * it + 1, a.err, &s_ok)) return;
    }
}

// ---- the FP32 CUDA-core kernel's sums (PFLBM_MLP_SIMT=1)
// Sums the block gradients (fixed order, FP64) into grad[0..kMlpParams]
// (the last entry is the loss sum).
__global__ void k_grad_sum(const float *__restrict__ gpart, int nblocks, double *__restrict__ grad) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > kMlpParams) return;
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += gpart[size_t(b) * (kMlpParams + 1) + p];
    grad[p] = s;
}

// Adam on the mean minibatch gradient; loss_log[iter] = mean minibatch loss.
__global__ void k_adam(float *__restrict__ blob, float *__restrict__ m, float *__restrict__ v,
                       const float *__restrict__ gpart, int nblocks, float inv_count, float lr, float beta1,
                       float beta2, float eps, float c1, float c2, double *__restrict__ loss_log, int iter) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > kMlpParams) return;
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += gpart[size_t(b) * (kMlpParams + 1) + p];
    if (p == kMlpParams) {
        loss_log[iter] = s * inv_count;
        return;
    }
    const float g = float(s) * inv_count;
    adam_update(g, lr, beta1, beta2, eps, c1, c2, m[p], v[p], blob[p]);
}

// Forward only: FP64 loss sum per block. A thread evaluates two samples at a
// time with packed FP32x2 arithmetic, the weights in shared memory twice side
// by side so that one 16-byte broadcast feeds two packed multiply-adds: the
// one-sample form issued a shared load per multiply-add and spilled its
// activations (255 registers). Each sample rounds as mlp_nu_t does. 2^20
// samples: 376 -> 130 us.
constexpr int kLossThreads = 128;
__global__ void __launch_bounds__(kLossThreads, 4) k_mlp_loss(const float *__restrict__ blob, const float *__restrict__ X,
                                                           const float *__restrict__ Y, uint64_t n,
                                                           double *__restrict__ partial) {
    using pflbm::V2;
    __shared__ __align__(16) float2 w[kMlpBlob];
    for (int i = threadIdx.x; i < kMlpBlob; i += kLossThreads) w[i] = make_float2(blob[i], blob[i]);
    __syncthreads();
    auto w2 = [&](int i, V2 &a, V2 &b) {  // weights i and i + 1, i even
        const float4 v = *reinterpret_cast<const float4 *>(&w[i]);
        a = V2(v.x, v.y);
        b = V2(v.z, v.w);
    };
    auto silu2 = [](V2 a) { return V2(pflbm::silu_d<float>(a.v.x), pflbm::silu_d<float>(a.v.y)); };
    static_assert(pflbm::kMlpW1 % 2 == 0 && pflbm::kMlpW2 % 2 == 0, "pairs of weights");
    const float out_scale = w[pflbm::kMlpOutScale].x;
    double acc = 0.0;
    const uint64_t pairs = (n + 1) / 2;
    for (uint64_t k = blockIdx.x * uint64_t(kLossThreads) + threadIdx.x; k < pairs;
         k += uint64_t(gridDim.x) * kLossThreads) {
        asm volatile("" ::: "memory");  // keeps the weight loads inside the loop (hoisted, they spill)
        const bool second = 2 * k + 1 < n;
        const float4 *xa = reinterpret_cast<const float4 *>(X + 2 * k * kMlpIn), *xb = second ? xa + 2 : xa;
        const float4 a0 = xa[0], a1 = xa[1], b0 = xb[0], b1 = xb[1];
        V2 xn[kMlpIn] = {V2(a0.x, b0.x), V2(a0.y, b0.y), V2(a0.z, b0.z), V2(a0.w, b0.w),
                         V2(a1.x, b1.x), V2(a1.y, b1.y), V2(a1.z, b1.z), V2(a1.w, b1.w)};
#pragma unroll
        for (int q = 0; q < kMlpIn; ++q)
            xn[q] = (xn[q] - V2(w[pflbm::kMlpMean + q])) * V2(w[pflbm::kMlpInvScale + q]);
        V2 h1[kMlpH];
#pragma unroll
        for (int i = 0; i < kMlpH; ++i) {
            V2 s(w[pflbm::kMlpB1 + i]), wa, wb;
#pragma unroll
            for (int q = 0; q < kMlpIn; q += 2) {
                w2(pflbm::kMlpW1 + i * kMlpIn + q, wa, wb);
                s = pflbm::fma2(wb, xn[q + 1], pflbm::fma2(wa, xn[q], s));
            }
            h1[i] = silu2(s);
        }
        V2 z(w[pflbm::kMlpB3]);
#pragma unroll 2
        for (int j = 0; j < kMlpH; ++j) {
            V2 s(w[pflbm::kMlpB2 + j]), wa, wb;
#pragma unroll
            for (int i = 0; i < kMlpH; i += 2) {
                w2(pflbm::kMlpW2 + j * kMlpH + i, wa, wb);
                s = pflbm::fma2(wb, h1[i + 1], pflbm::fma2(wa, h1[i], s));
            }
            z = pflbm::fma2(V2(w[pflbm::kMlpW3 + j]), silu2(s), z);
        }
        const float ra = (out_scale * pflbm::softplus_d<float>(z.v.x) - Y[2 * k]) / out_scale;
        acc += double(ra) * ra;
        if (second) {
            const float rb = (out_scale * pflbm::softplus_d<float>(z.v.y) - Y[2 * k + 1]) / out_scale;
            acc += double(rb) * rb;
        }
    }
    __shared__ double sh[kLossThreads];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int st = kLossThreads / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

}  // namespace

// ------------------------------------------------------------- object
struct pflbm_closure {
    int device = 0;
    cudaStream_t stream = nullptr;
    uint64_t cap = 0, n = 0;
    float *X = nullptr, *Y = nullptr;
    float *blob = nullptr, *m = nullptr, *v = nullptr;
    float *gpart = nullptr;  // per-block gradients of the CUDA-core kernel
    int gpart_blocks = 0;
    double *gsum = nullptr;  // per-CTA gradient sums of the tensor-core kernels
    int grad_ctas = 0, train_ctas = 0;  // resident CTAs of the gradient and the training kernel
    unsigned int *sync = nullptr;  // grid barrier count and error word of the training kernel
    double *grad = nullptr, *partial = nullptr, *loss_log = nullptr;
    int loss_log_cap = 0;
    float *coarse = nullptr;
    uint64_t coarse_cap = 0;
    double *width_part = nullptr;           // per-block interface sums of a snapshot
    double width_sum[4] = {0, 0, 0, 0};     // phi(1-phi), |grad phi|: filtered coarse, fine
    uint64_t adam_t = 0;
    bool have_params = false;
    std::vector<float> host_blob = std::vector<float>(kMlpBlob, 0.0f);

    ~pflbm_closure() {
        cudaSetDevice(device);
        void *ptrs[] = {X, Y, blob, m, v, gpart, gsum, sync, grad, partial, loss_log, coarse, width_part};
        for (void *p : ptrs)
            if (p) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

int ensure_gpart(pflbm_closure *c, int blocks) {
    if (blocks <= c->gpart_blocks) return PFLBM_OK;
    if (c->gpart) cudaFree(c->gpart);
    c->gpart = nullptr;
    c->gpart_blocks = 0;
    cudaError_t e = cudaMalloc(&c->gpart, sizeof(float) * size_t(blocks) * (kMlpParams + 1));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc (gradient partials)");
    c->gpart_blocks = blocks;
    return PFLBM_OK;
}

int upload_blob(pflbm_closure *c) {
    cudaError_t e = cudaMemcpyAsync(c->blob, c->host_blob.data(), sizeof(float) * kMlpBlob, cudaMemcpyHostToDevice,
                                    c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    return e == cudaSuccess ? PFLBM_OK : cuda_fail(e, "closure blob upload");
}

int download_blob(pflbm_closure *c) {
    cudaError_t e = cudaMemcpyAsync(c->host_blob.data(), c->blob, sizeof(float) * kMlpBlob, cudaMemcpyDeviceToHost,
                                    c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    return e == cudaSuccess ? PFLBM_OK : cuda_fail(e, "closure blob download");
}

size_t act_bytes() { return sizeof(Act); }

// Gradients by the tensor-core kernels, or with PFLBM_MLP_SIMT=1 by the FP32
// CUDA-core kernel (exact FP32 products, for checks against the FP64 oracle at
// FP32 rounding).
bool use_simt_grad() {
    const char *e = std::getenv("PFLBM_MLP_SIMT");
    return e && e[0] == '1';
}

void launch_grad_simt(pflbm_closure *c, int blocks, int mode, uint64_t seed, uint64_t iter, uint64_t count) {
    k_mlp_grad<<<blocks, kSB, act_bytes(), c->stream>>>(c->blob, c->X, c->Y, c->n, mode, seed, iter, count, c->gpart);
}

// Iterations it0 .. it0 + k - 1 of a training call in one cooperative launch:
// one CTA per block and at least one per 16 parameters, as far as they are
// all resident.
cudaError_t launch_train(pflbm_closure *c, TrainArgs &a) {
    const int grid = std::min(std::max(kSumCtas, a.blocks), c->train_ctas);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = pflbm::launch_grid(dim3(grid));
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = kTcSmem;
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_mlp_train, a);
}

}  // namespace

extern "C" {

int pflbm_closure_create(int32_t device, uint64_t max_samples, pflbm_closure **out) {
    if (!out || max_samples == 0) return fail(PFLBM_ERR_INVALID_ARG, "bad argument");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fail(PFLBM_ERR_CUDA, "no CUDA device");
    }
    if (device < 0 || device >= ndev) return fail(PFLBM_ERR_INVALID_ARG, "device out of range");
    std::unique_ptr<pflbm_closure> c(new (std::nothrow) pflbm_closure());
    if (!c) return fail(PFLBM_ERR_OUT_OF_MEMORY, "closure handle");
    c->device = device;
    cudaSetDevice(device);
    c->cap = max_samples;
    cudaError_t e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamCreate");
    if (cudaMalloc(&c->X, sizeof(float) * kMlpIn * max_samples) != cudaSuccess ||
        cudaMalloc(&c->Y, sizeof(float) * max_samples) != cudaSuccess ||
        cudaMalloc(&c->blob, sizeof(float) * kMlpBlob) != cudaSuccess ||
        cudaMalloc(&c->m, sizeof(float) * kMlpParams) != cudaSuccess ||
        cudaMalloc(&c->v, sizeof(float) * kMlpParams) != cudaSuccess ||
        cudaMalloc(&c->grad, sizeof(double) * (kMlpParams + 1)) != cudaSuccess ||
        cudaMalloc(&c->partial, sizeof(double) * kLossBlocks * 18) != cudaSuccess ||
        cudaMalloc(&c->sync, 2 * sizeof(unsigned int)) != cudaSuccess ||
        cudaMalloc(&c->width_part, sizeof(double) * kMakeBlocks * 4) != cudaSuccess) {
        cudaGetLastError();
        return fail(PFLBM_ERR_OUT_OF_MEMORY, "closure buffers");
    }
    if (cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, int(act_bytes())) != cudaSuccess)
        return cuda_fail(cudaGetLastError(), "k_mlp_grad shared memory");
    if (cudaFuncSetAttribute(k_mlp_grad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess)
        return cuda_fail(cudaGetLastError(), "gradient kernel shared memory");
    // both kernels run at most as many CTAs as are resident at once
    int sms = 0, grad = 0, train = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&grad, k_mlp_grad_tc, kTcThreads, kTcSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&train, k_mlp_train, kTcThreads, kTcSmem) != cudaSuccess ||
        grad < 1 || train < 1)
        return cuda_fail(cudaGetLastError(), "training kernel occupancy");
    c->grad_ctas = sms * grad;
    c->train_ctas = sms * train;
    if (cudaMalloc(&c->gsum, sizeof(double) * size_t(std::max(c->grad_ctas, c->train_ctas)) * kTcPart) != cudaSuccess) {
        cudaGetLastError();
        return fail(PFLBM_ERR_OUT_OF_MEMORY, "closure buffers");
    }
    *out = c.release();
    return PFLBM_OK;
}

int pflbm_closure_destroy(pflbm_closure *c) {
    delete c;
    return PFLBM_OK;
}

int pflbm_closure_num_samples(const pflbm_closure *c, uint64_t *n) {
    if (!c || !n) return fail(PFLBM_ERR_INVALID_ARG, "null argument");
    *n = c->n;
    return PFLBM_OK;
}

int pflbm_closure_add_snapshot(pflbm_closure *c, pflbm_sim *fine, int32_t stride, uint64_t *added) {
    if (!c || !fine || stride < 1) return fail(PFLBM_ERR_INVALID_ARG, "bad argument");
    pflbm::SimView v{};
    if (int rc = pflbm::sim_view(fine, v)) return rc;
    if (v.real_bytes != 4) return fail(PFLBM_ERR_UNSUPPORTED, "training snapshots need an FP32 or 16-bit storage run");
    if (v.device != c->device) return fail(PFLBM_ERR_INVALID_ARG, "simulation and closure are on different devices");
    if (v.nx % 2 || v.ny % 2 || v.nz % 2 || v.nx < 16 || v.ny < 16 || v.nz < 16)
        return fail(PFLBM_ERR_INVALID_ARG, "fine grid extents must be even and >= 16");
    cudaSetDevice(c->device);
    const int nxc = int(v.nx / 2), nyc = int(v.ny / 2), nzc = int(v.nz / 2);
    const uint64_t Nc = uint64_t(nxc) * nyc * nzc;
    if (c->coarse_cap < Nc) {
        if (c->coarse) cudaFree(c->coarse);
        c->coarse = nullptr;
        c->coarse_cap = 0;
        if (cudaMalloc(&c->coarse, sizeof(float) * kCoarseFields * Nc) != cudaSuccess) {
            cudaGetLastError();
            return fail(PFLBM_ERR_OUT_OF_MEMORY, "closure coarse scratch");
        }
        c->coarse_cap = Nc;
    }
    // sample lattice: i = i0, i0 + stride, ... within [2, nxc-3]
    const int i0 = ((2 + stride - 1) / stride) * stride, j0 = i0;
    const int ni = i0 > nxc - 3 ? 0 : (nxc - 3 - i0) / stride + 1;
    const int nj = j0 > nyc - 3 ? 0 : (nyc - 3 - j0) / stride + 1;
    const uint64_t count = uint64_t(ni) * nj * uint64_t(nzc - 4);
    if (c->n + count > c->cap)
        return fail(PFLBM_ERR_INVALID_ARG, "closure sample capacity exceeded (" + std::to_string(c->n + count) + " > " +
                                               std::to_string(c->cap) + ")");
    // the fine run's analysis ran on its own stream, which sim_view synchronised
    const dim3 fg((nxc + kFilterX - 1) / kFilterX, (nyc + kFilterY - 1) / kFilterY,
                  (nzc + kFilterPlanes - 1) / kFilterPlanes);
    k_filter_restrict<<<fg, dim3(kFilterX, kFilterY), 0, c->stream>>>(
        static_cast<const float *>(v.macro), v.N, int(v.nx), int(v.ny), int(v.nz), nxc, nyc, nzc, c->coarse);
    k_make_samples<<<kMakeBlocks, kMakeThreads, 0, c->stream>>>(
        c->coarse, nxc, nyc, nzc, stride, float(v.tau_water), float(v.tau_oil), i0, ni, j0, nj, c->X, c->Y, c->n,
        static_cast<const float *>(v.macro), v.N, int(v.nx), int(v.ny), c->width_part);
    std::vector<double> wp(size_t(kMakeBlocks) * 4);
    cudaError_t e = cudaMemcpyAsync(wp.data(), c->width_part, sizeof(double) * wp.size(), cudaMemcpyDeviceToHost,
                                    c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "closure snapshot");
    for (int b = 0; b < kMakeBlocks; ++b)
        for (int q = 0; q < 4; ++q) c->width_sum[q] += wp[size_t(b) * 4 + q];
    c->n += count;
    if (added) *added = count;
    return PFLBM_OK;
}

int pflbm_closure_interface_scale(const pflbm_closure *c, double *gamma_scale, double *width_fine,
                                   double *width_filtered) {
    if (!c || !gamma_scale) return fail(PFLBM_ERR_INVALID_ARG, "null argument");
    const double *w = c->width_sum;
    if (!(w[0] > 0.0 && w[1] > 0.0 && w[2] > 0.0 && w[3] > 0.0))
        return fail(PFLBM_ERR_STATE, "no interface in the snapshots added so far");
    const double wc = 4.0 * w[0] / w[1], wf = 4.0 * w[2] / w[3];
    *gamma_scale = wf / wc;
    if (width_fine) *width_fine = wf;
    if (width_filtered) *width_filtered = wc;
    return PFLBM_OK;
}

int pflbm_closure_get_samples(pflbm_closure *c, uint64_t first, uint64_t count, float *host_x, float *host_y) {
    if (!c || (!host_x && !host_y) || first + count > c->n) return fail(PFLBM_ERR_INVALID_ARG, "bad sample range");
    cudaSetDevice(c->device);
    cudaError_t e = cudaSuccess;
    if (host_x)
        e = cudaMemcpy(host_x, c->X + first * kMlpIn, sizeof(float) * kMlpIn * count, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && host_y) e = cudaMemcpy(host_y, c->Y + first, sizeof(float) * count, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? PFLBM_OK : cuda_fail(e, "sample readback");
}

int pflbm_closure_set_samples(pflbm_closure *c, const float *host_x, const float *host_y, uint64_t count) {
    if (!c || !host_x || !host_y || count > c->cap) return fail(PFLBM_ERR_INVALID_ARG, "bad argument");
    cudaSetDevice(c->device);
    cudaError_t e = cudaMemcpy(c->X, host_x, sizeof(float) * kMlpIn * count, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(c->Y, host_y, sizeof(float) * count, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "sample upload");
    c->n = count;
    return PFLBM_OK;
}

int pflbm_closure_init_params(pflbm_closure *c, uint32_t seed) {
    if (!c) return fail(PFLBM_ERR_INVALID_ARG, "null closure");
    if (c->n == 0) return fail(PFLBM_ERR_STATE, "no training samples");
    cudaSetDevice(c->device);
    const int blocks = 304;
    k_stats<<<blocks, 256, 0, c->stream>>>(c->X, c->Y, c->n, c->partial);
    std::vector<double> part(size_t(blocks) * 18);
    cudaError_t e = cudaMemcpyAsync(part.data(), c->partial, sizeof(double) * part.size(), cudaMemcpyDeviceToHost,
                                    c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "closure statistics");
    double tot[18] = {0};
    for (int b = 0; b < blocks; ++b)
        for (int f = 0; f < 18; ++f) tot[f] += part[size_t(b) * 18 + f];
    const double n = double(c->n);
    std::vector<float> &w = c->host_blob;
    std::fill(w.begin(), w.end(), 0.0f);
    for (int k = 0; k < kMlpIn; ++k) {
        const double mean = tot[k] / n;
        const double var = std::max(tot[8 + k] / n - mean * mean, 0.0);
        w[pflbm::kMlpMean + k] = float(mean);
        w[pflbm::kMlpInvScale + k] = var > 1e-30 ? float(1.0 / std::sqrt(var)) : 1.0f;
    }
    const double ymean = tot[16] / n, yrms = std::sqrt(std::max(tot[17] / n, 0.0));
    const double out_scale = yrms > 1e-30 ? yrms : 1.0;
    w[pflbm::kMlpOutScale] = float(out_scale);
    w[pflbm::kMlpStrength] = 1.0f;
    // Glorot-uniform weights from a counter hash, zero biases; b3 puts the
    // initial output at the mean target
    auto uni = [&](uint64_t k) { return double(mix64(uint64_t(seed) * 0x9E3779B97F4A7C15ull + k) >> 11) * 0x1.0p-53; };
    const double l1 = std::sqrt(6.0 / (kMlpIn + kMlpH)), l2 = std::sqrt(6.0 / (2 * kMlpH)),
                 l3 = std::sqrt(6.0 / (kMlpH + 1));
    for (int p = 0; p < kMlpH * kMlpIn; ++p) w[pflbm::kMlpW1 + p] = float(l1 * (2.0 * uni(p) - 1.0));
    for (int p = 0; p < kMlpH * kMlpH; ++p) w[pflbm::kMlpW2 + p] = float(l2 * (2.0 * uni(10000 + p) - 1.0));
    for (int p = 0; p < kMlpH; ++p) w[pflbm::kMlpW3 + p] = float(l3 * (2.0 * uni(20000 + p) - 1.0));
    const double t0 = std::max(ymean / out_scale, 1e-3);
    w[pflbm::kMlpB3] = float(t0 > 20.0 ? t0 : std::log(std::expm1(t0)));
    if (int rc = upload_blob(c)) return rc;
    cudaMemsetAsync(c->m, 0, sizeof(float) * kMlpParams, c->stream);
    cudaMemsetAsync(c->v, 0, sizeof(float) * kMlpParams, c->stream);
    e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "closure init");
    c->adam_t = 0;
    c->have_params = true;
    return PFLBM_OK;
}

int pflbm_closure_get_blob(pflbm_closure *c, float *host_blob) {
    if (!c || !host_blob) return fail(PFLBM_ERR_INVALID_ARG, "null argument");
    cudaSetDevice(c->device);
    if (int rc = download_blob(c)) return rc;
    std::memcpy(host_blob, c->host_blob.data(), sizeof(float) * kMlpBlob);
    return PFLBM_OK;
}

int pflbm_closure_set_blob(pflbm_closure *c, const float *host_blob) {
    if (!c || !host_blob) return fail(PFLBM_ERR_INVALID_ARG, "null argument");
    cudaSetDevice(c->device);
    std::memcpy(c->host_blob.data(), host_blob, sizeof(float) * kMlpBlob);
    if (int rc = upload_blob(c)) return rc;
    cudaMemsetAsync(c->m, 0, sizeof(float) * kMlpParams, c->stream);
    cudaMemsetAsync(c->v, 0, sizeof(float) * kMlpParams, c->stream);
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "closure set blob");
    c->adam_t = 0;
    c->have_params = true;
    return PFLBM_OK;
}

int pflbm_closure_gradient(pflbm_closure *c, uint64_t count, double *host_grad, double *loss_sum) {
    if (!c || !host_grad || count == 0 || count > c->n) return fail(PFLBM_ERR_INVALID_ARG, "bad argument");
    if (!c->have_params) return fail(PFLBM_ERR_STATE, "closure parameters not initialised");
    cudaSetDevice(c->device);
    const int blocks = int((count + kSB - 1) / kSB);
    if (use_simt_grad()) {
        if (int rc = ensure_gpart(c, blocks)) return rc;
        launch_grad_simt(c, blocks, 0, 0, 0, count);
        k_grad_sum<<<(kMlpParams + 1 + 255) / 256, 256, 0, c->stream>>>(c->gpart, blocks, c->grad);
    } else {
        const int ctas = std::min(blocks, c->grad_ctas);
        k_mlp_grad_tc<<<ctas, kTcThreads, kTcSmem, c->stream>>>(c->blob, c->X, c->Y, c->n, count, blocks, c->gsum);
        k_grad_rows<<<kSumCtas, kTcThreads, 0, c->stream>>>(c->gsum, ctas, c->grad);
    }
    std::vector<double> g(kMlpParams + 1);
    cudaError_t e = cudaMemcpyAsync(g.data(), c->grad, sizeof(double) * g.size(), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "closure gradient");
    std::memcpy(host_grad, g.data(), sizeof(double) * kMlpParams);
    if (loss_sum) *loss_sum = g[kMlpParams];
    return PFLBM_OK;
}

int pflbm_closure_train(pflbm_closure *c, int32_t iterations, int32_t batch, float lr, uint32_t seed,
                        double *loss_history) {
    if (!c || iterations < 1 || batch < 1) return fail(PFLBM_ERR_INVALID_ARG, "bad argument");
    if (!c->have_params) return fail(PFLBM_ERR_STATE, "closure parameters not initialised");
    if (c->n == 0) return fail(PFLBM_ERR_STATE, "no training samples");
    cudaSetDevice(c->device);
    const int blocks = int((int64_t(batch) + kSB - 1) / kSB);
    const bool simt = use_simt_grad();
    if (simt)
        if (int rc = ensure_gpart(c, blocks)) return rc;
    if (c->loss_log_cap < iterations) {
        if (c->loss_log) cudaFree(c->loss_log);
        c->loss_log = nullptr;
        c->loss_log_cap = 0;
        if (cudaMalloc(&c->loss_log, sizeof(double) * iterations) != cudaSuccess) {
            cudaGetLastError();
            return fail(PFLBM_ERR_OUT_OF_MEMORY, "loss log");
        }
        c->loss_log_cap = iterations;
    }
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    auto correction = [](float beta, uint64_t t) { return float(1.0 - std::pow(double(beta), double(t))); };
    if (simt) {
        for (int it = 0; it < iterations; ++it) {
            const uint64_t t = ++c->adam_t;
            launch_grad_simt(c, blocks, 1, seed, t, uint64_t(batch));
            k_adam<<<(kMlpParams + 1 + 255) / 256, 256, 0, c->stream>>>(
                c->blob, c->m, c->v, c->gpart, blocks, 1.0f / float(batch), lr, beta1, beta2, eps,
                correction(beta1, t), correction(beta2, t), c->loss_log, it);
        }
    } else {
        TrainArgs a{};
        a.blob = c->blob, a.m = c->m, a.v = c->v, a.X = c->X, a.Y = c->Y;
        a.n = c->n, a.seed = seed, a.count = uint64_t(batch), a.blocks = blocks;
        a.inv_count = 1.0f / float(batch), a.lr = lr, a.beta1 = beta1, a.beta2 = beta2, a.eps = eps;
        a.gsum = c->gsum, a.loss_log = c->loss_log, a.arrived = c->sync, a.err = c->sync + 1;
        cudaMemsetAsync(c->sync, 0, 2 * sizeof(unsigned int), c->stream);
        int launched = 0;  // iterations; they count when they have run
        cudaError_t le = cudaSuccess;
        while (launched < iterations) {
            a.iterations = std::min(kTrainChunk, iterations - launched);
            a.iter0 = c->adam_t + launched + 1;
            a.log0 = launched;
            for (int k = 0; k < a.iterations; ++k) {
                a.c1[k] = correction(beta1, a.iter0 + k);
                a.c2[k] = correction(beta2, a.iter0 + k);
            }
            if (launched > 0) cudaMemsetAsync(c->sync, 0, sizeof(unsigned int), c->stream);
            le = launch_train(c, a);
            if (le != cudaSuccess) break;  // what was launched before still counts
            launched += a.iterations;
        }
        cudaError_t e = cudaStreamSynchronize(c->stream);
        unsigned int w = 0;
        if (e == cudaSuccess) e = cudaMemcpy(&w, c->sync + 1, sizeof w, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess || w != 0) c->have_params = false;  // of no known iteration
        if (e != cudaSuccess) return cuda_fail(e, "closure training");
        if (w)
            return fail(PFLBM_ERR_DEVICE,
                        "the training kernel gave up waiting at its grid barrier; set or initialise the parameters again");
        c->adam_t += launched;
        if (le != cudaSuccess) return cuda_fail(le, "training launch");
    }
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "closure training");
    if (loss_history) {
        e = cudaMemcpy(loss_history, c->loss_log, sizeof(double) * iterations, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return cuda_fail(e, "loss history");
    }
    return download_blob(c);
}

int pflbm_closure_loss(pflbm_closure *c, double *mean_loss) {
    if (!c || !mean_loss) return fail(PFLBM_ERR_INVALID_ARG, "null argument");
    if (!c->have_params || c->n == 0) return fail(PFLBM_ERR_STATE, "no parameters or samples");
    cudaSetDevice(c->device);
    k_mlp_loss<<<kLossBlocks, kLossThreads, 0, c->stream>>>(c->blob, c->X, c->Y, c->n, c->partial);
    std::vector<double> part(kLossBlocks);
    cudaError_t e = cudaMemcpyAsync(part.data(), c->partial, sizeof(double) * kLossBlocks, cudaMemcpyDeviceToHost,
                                    c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "closure loss");
    double s = 0.0;
    for (double p : part) s += p;
    *mean_loss = s / double(c->n);
    return PFLBM_OK;
}

}  // extern "C"

// reduce.cuh - block reduction of the FP64 diagnostics rows (phi mass, rho
// mass, momentum, max |u|, inside/outside rho and counts, non-finite count)
// with warp shuffles.
#pragma once
#include <cuda_runtime.h>

#include "widen.cuh"

namespace pflbm {

constexpr int RED_FIELDS = 12;  // phi, rho, rho ux, rho uy, rho uz, max |u|^2, rho_in, n_in, rho_out, n_out, nonfinite, spare
constexpr int RED_MAX_SLOT = 5; // max |u|^2 (combined by max; every other slot by sum)

// A thread's sums over its nodes. FP64 is the scarce unit (about 2 lanes per
// clock and SM): what needs no FP64 is kept off it. The counts are integers,
// float fields are classified as floats (phi > 0.9 and phi < 0.1 select the
// same floats against 0.9f and 0.1f), and the square root is taken of the
// largest |u|^2 only, which gives the largest root (the root is monotone).
// Floats are widened on the integer units. With the 64-bit divisions per node
// gone as well, 128^3 nodes and the final pass: 222 -> 73 us.
struct RedAcc {
    double phi = 0.0, rho = 0.0, mx = 0.0, my = 0.0, mz = 0.0, u2 = 0.0, rho_in = 0.0, rho_out = 0.0;
    unsigned int n_in = 0u, n_out = 0u, bad = 0u;

    template <class T>
    __device__ __forceinline__ void add(T r, T ux, T uy, T uz, T p) {
        if (!isfinite(p) || !isfinite(r) || !isfinite(ux) || !isfinite(uy) || !isfinite(uz)) {
            ++bad;
            return;
        }
        const T in[5] = {r, ux, uy, uz, p};
        double wide[5];
        if constexpr (sizeof(T) == 4) {
            widen_all(in, wide);
        } else {
#pragma unroll
            for (int k = 0; k < 5; ++k) wide[k] = in[k];
        }
        const double dr = wide[0], dx = wide[1], dy = wide[2], dz = wide[3];
        phi += wide[4];
        rho += dr;
        mx = fma(dr, dx, mx);
        my = fma(dr, dy, my);
        mz = fma(dr, dz, mz);
        const double s = fma(dz, dz, fma(dy, dy, dx * dx));
        if (s > u2) u2 = s;
        if (p > T(0.9)) {
            rho_in += dr;
            ++n_in;
        }
        if (p < T(0.1)) {
            rho_out += dr;
            ++n_out;
        }
    }
    __device__ __forceinline__ void row(double (&acc)[RED_FIELDS]) const {
        const double v[RED_FIELDS] = {phi, rho, mx, my, mz, u2, rho_in, double(n_in), rho_out, double(n_out), double(bad), 0.0};
#pragma unroll
        for (int f = 0; f < RED_FIELDS; ++f) acc[f] = v[f];
    }
};

__device__ __forceinline__ double red_combine(int f, double a, double b) {
    return f == RED_MAX_SLOT ? fmax(a, b) : a + b;
}

// Reduces each thread's `acc` over the block (NTHREADS, a multiple of 32):
// a shuffle tree inside every warp, then the warps' results, in warp order,
// by a shuffle tree in the first warp. Thread 0 writes the row to `out`.
// Every value is >= 0 in the max slot, so 0 is the identity of both
// operations. Deterministic: the order of combination is fixed.
template <int NTHREADS>
__device__ __forceinline__ void block_reduce_row(double (&acc)[RED_FIELDS], double *out) {
    static_assert(NTHREADS % 32 == 0 && NTHREADS <= 1024, "block size");
    constexpr int NW = NTHREADS / 32;
    __shared__ double s_warp[NW][RED_FIELDS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int f = 0; f < RED_FIELDS; ++f) {
        double v = acc[f];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = red_combine(f, v, __shfl_down_sync(0xffffffffu, v, o));
        if (lane == 0) s_warp[warp][f] = v;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int f = 0; f < RED_FIELDS; ++f) {
            double v = lane < NW ? s_warp[lane][f] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = red_combine(f, v, __shfl_down_sync(0xffffffffu, v, o));
            if (lane == 0) out[f] = v;
        }
    }
}

// The total of `n` rows in slot f, by the calling warp (lane-strided, then a
// shuffle tree; lane 0 has it); the max slot becomes max |u|. One thread per
// slot took 71 us for 608 rows, a warp per slot takes 9.
constexpr int RED_FINAL_THREADS = 32 * RED_FIELDS;
__device__ __forceinline__ double red_total(const double *rows, int n, int f) {
    double s = 0.0;
#pragma unroll 4
    for (int b = int(threadIdx.x) & 31; b < n; b += 32) s = red_combine(f, s, rows[size_t(b) * RED_FIELDS + f]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = red_combine(f, s, __shfl_down_sync(0xffffffffu, s, o));
    return f == RED_MAX_SLOT ? sqrt(s) : s;
}

}  // namespace pflbm

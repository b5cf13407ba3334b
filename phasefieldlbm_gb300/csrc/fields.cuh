// fields.cuh - initial conditions, ghost-shell readback, vorticity and the FP64
// diagnostics reductions.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "boundary.cuh"
#include "lattice.cuh"
#include "params.cuh"
#include "reduce.cuh"
#include "tile.h"

namespace pflbm {

// ------------------------------------------------------------ init
// Initial macroscopic fields into the analysis cache (rho, u, phi), every
// node: setInitialDensity + setJet / setDroplet (src/initialConditions.cu:33-99).
struct InitGeom {
    int jet;
    float droplet_x_stretch;
    float center_z;
    int radius;
    float interface_width;
    float init_noise;
};

template <class T>
__global__ void k_init_fields(const Params<T> p, const InitGeom g, T *macro) {
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const uint64_t N = p.Nd;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z * blockDim.z + threadIdx.z;
    if (x >= nx || y >= ny || z >= nz) return;
    const uint64_t i = static_cast<uint64_t>(x) + static_cast<uint64_t>(nx) * (y + static_cast<uint64_t>(ny) * z);
    for (int s = 0; s < M_COUNT; ++s) macro[s * N + i] = T(0);
    macro[M_RHO * N + i] = T(1);
    if (g.jet) {
        if (z == 0 && in_disc<T>(p, x, y)) {
            macro[M_PHI * N + i] = T(1);
            macro[M_UZ * N + i] = p.u_inf;
        }
    } else if (x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2 && z >= 1 && z <= nz - 2) {
        const T dx = (static_cast<T>(x) - p.center_x) / static_cast<T>(g.droplet_x_stretch);
        const T dy = static_cast<T>(y) - p.center_y;
        const T dz = static_cast<T>(z) - static_cast<T>(g.center_z);
        const T L2 = sqrt(dx * dx + dy * dy + dz * dz);
        const T arg = static_cast<T>((static_cast<double>(g.radius) - static_cast<double>(L2)) / static_cast<double>(g.interface_width));
        macro[M_PHI * N + i] = T(0.5) + T(0.5) * tanh(T(2) * arg);
        if (g.init_noise != 0.0f) {
            macro[M_UX * N + i] = static_cast<T>(g.init_noise * init_noise_value(p.seed, 0, x, y, z));
            macro[M_UY * N + i] = static_cast<T>(g.init_noise * init_noise_value(p.seed, 1, x, y, z));
            macro[M_UZ * N + i] = static_cast<T>(g.init_noise * init_noise_value(p.seed, 2, x, y, z));
        }
    }
}

// setDistros (src/initialConditions.cu:101-138) expressed in the pull
// layout: f^0_q(X) = feq_q(rho_X, u_X) is written to slot X - c_q of both
// ping-pong buffers; phi^0 = sum_q geq_q (computePhase of step 0); ghost phi
// takes the initial ghost values.
template <int QQ, bool JET, class S>
__global__ void k_init_distros(const Params<typename Store<S>::T> p, S *fa, S *fb, typename Store<S>::T *phia,
                               typename Store<S>::T *phib, const typename Store<S>::T *macro) {
    using T = typename Store<S>::T;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const uint64_t N = p.N, Nd = p.Nd;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z * blockDim.z + threadIdx.z;
    if (x >= nx || y >= ny || z >= nz) return;
    const uint64_t i = static_cast<uint64_t>(x) + static_cast<uint64_t>(nx) * (y + static_cast<uint64_t>(ny) * z);
    const uint64_t ip = static_cast<uint64_t>(x) + static_cast<uint64_t>(p.px) * (y + static_cast<uint64_t>(ny) * z);
    const T phi0 = macro[M_PHI * Nd + i];
    if (x < 1 || x > nx - 2 || y < 1 || y > ny - 2 || z < 1 || z > nz - 2) {
        phia[ip] = phi0;
        phib[ip] = phi0;
        return;
    }
    const T rho = macro[M_RHO * Nd + i], ux = macro[M_UX * Nd + i], uy = macro[M_UY * Nd + i], uz = macro[M_UZ * Nd + i];
#pragma unroll
    for (int q = 0; q < QQ; ++q) {
        const T v = feq_q<QQ, T>(q, rho, ux, uy, uz);
        const int64_t off = kCX[q] + static_cast<int64_t>(kCY[q]) * p.px + static_cast<int64_t>(kCZ[q]) * static_cast<int64_t>(p.plane);
        Store<S>::store(fa, q * N + ip - off, v, static_cast<T>(1.0 / weight<QQ>(q)));
        Store<S>::store(fb, q * N + ip - off, v, static_cast<T>(1.0 / weight<QQ>(q)));
    }
    T s = T(0);
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        const T w = static_cast<T>(weight7(q));
        s += w * phi0 * (T(1) + T(4) * cdot<T>(kCX[q], kCY[q], kCZ[q], ux, uy, uz));
    }
    phia[ip] = s;
    phib[ip] = phi0;
}

// Ghost-shell values of the reference's arrays after a step (analysis):
// rho = 1 and zeros (FieldAllocate memset + setInitialDensity), inlet ghost
// plane from the inflow, outlet ghost plane copied from nz-2. One thread per
// node of the shell (a launch over all nodes spent 80 us on 128x128x512
// finding the 3% that are ghosts); `full`: all 18 arrays, else those of
// MODE_ANALYSIS_BASE.
__host__ __device__ inline uint64_t shell_nodes(uint64_t nx, uint64_t ny, uint64_t nz) {
    return 2 * nx * ny + (nz - 2) * (2 * nx + 2 * (ny - 2));
}
template <class T>
__global__ void __launch_bounds__(256) k_analysis_ghosts(const Params<T> p, int jet, uint32_t t, T *macro, bool full) {
    const uint32_t nx = p.nx, ny = p.ny, nz = p.nz;
    const uint64_t N = p.Nd;
    const uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    if (k >= shell_nodes(nx, ny, nz)) return;
    // the planes z = 0 and nz-1, then per plane the rows y = 0 and ny-1 and
    // the columns x = 0 and nx-1
    uint32_t x, y, z;
    const uint64_t plane = uint64_t(nx) * ny;
    if (k < 2 * plane) {
        const uint32_t r = uint32_t(k < plane ? k : k - plane);
        z = k < plane ? 0 : nz - 1;
        x = r % nx;
        y = r / nx;
    } else {
        const uint32_t ring = 2 * nx + 2 * (ny - 2), s = uint32_t(k - 2 * plane);
        const uint32_t r = s % ring;
        z = 1 + s / ring;
        if (r < 2 * nx) {
            x = r < nx ? r : r - nx;
            y = r < nx ? 0 : ny - 1;
        } else {
            x = (r - 2 * nx) & 1 ? nx - 1 : 0;
            y = 1 + (r - 2 * nx) / 2;
        }
    }
    const uint64_t i = x + uint64_t(nx) * (y + uint64_t(ny) * z);
    T rho = T(1), ux = T(0), uy = T(0), uz = T(0), phi = T(0);
    if (jet && z == 0 && in_disc<T>(p, int(x), int(y))) {
        inflow_velocity<T>(p, x, y, t, ux, uy, uz);
        phi = T(1);
    } else if (jet && z == nz - 1 && x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2) {
        const uint64_t j = i - plane;
        rho = macro[M_RHO * N + j];
        ux = macro[M_UX * N + j];
        uy = macro[M_UY * N + j];
        uz = macro[M_UZ * N + j];
        phi = macro[M_PHI * N + j];
    }
    macro[M_RHO * N + i] = rho;
    macro[M_UX * N + i] = ux;
    macro[M_UY * N + i] = uy;
    macro[M_UZ * N + i] = uz;
    macro[M_PHI * N + i] = phi;
    macro[M_IND * N + i] = T(0);
    if (full)
        for (int s : {(int)M_PXX, (int)M_PYY, (int)M_PZZ, (int)M_PXY, (int)M_PXZ, (int)M_PYZ, (int)M_NX, (int)M_NY,
                      (int)M_NZ, (int)M_FX, (int)M_FY, (int)M_FZ})
            macro[s * N + i] = T(0);
}

// Vorticity by central differences, src/derivedFields/operators/vorticityFields.cuh:37-105.
template <class T>
__global__ void k_vorticity(const Params<T> p, const T *macro, T *vort) {
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const uint64_t N = p.Nd;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z * blockDim.z + threadIdx.z;
    if (x >= nx || y >= ny || z >= nz) return;
    const uint64_t i = static_cast<uint64_t>(x) + static_cast<uint64_t>(nx) * (y + static_cast<uint64_t>(ny) * z);
    T wx = T(0), wy = T(0), wz = T(0);
    if (x > 0 && x < nx - 1 && y > 0 && y < ny - 1 && z > 0 && z < nz - 1) {
        const T *ux = macro + M_UX * N, *uy = macro + M_UY * N, *uz = macro + M_UZ * N;
        const uint64_t sx = 1, sy = nx, sz = static_cast<uint64_t>(nx) * ny;
        const T h = T(0.5);
        const T duz_dy = h * (uz[i + sy] - uz[i - sy]);
        const T duy_dz = h * (uy[i + sz] - uy[i - sz]);
        const T dux_dz = h * (ux[i + sz] - ux[i - sz]);
        const T duz_dx = h * (uz[i + sx] - uz[i - sx]);
        const T duy_dx = h * (uy[i + sx] - uy[i - sx]);
        const T dux_dy = h * (ux[i + sy] - ux[i - sy]);
        wx = duz_dy - duy_dz;
        wy = dux_dz - duz_dx;
        wz = duy_dx - dux_dy;
    }
    vort[i] = wx;
    vort[N + i] = wy;
    vort[2 * N + i] = wz;
    vort[3 * N + i] = sqrt(wx * wx + wy * wy + wz * wz);
}

// FP64 diagnostics: per-block partial sums over interior nodes, then a
// single-block pass over the partials in fixed order (deterministic).
constexpr int RED_THREADS = 256;

template <class T>
__global__ void __launch_bounds__(RED_THREADS) k_reduce_partial(const Params<T> p, const T *macro, double *partial) {
    const uint32_t wx = p.nx - 2, wy = p.ny - 2;
    const uint64_t N = p.Nd, nint = uint64_t(wx) * wy * (p.nz - 2);
    const uint64_t first = blockIdx.x * uint64_t(RED_THREADS) + threadIdx.x, stride = uint64_t(gridDim.x) * RED_THREADS;
    RedAcc acc;
    // node k and the stride as (x, y, z) of the interior, carried on by
    // additions: no division per node
    uint32_t x = uint32_t(first % wx), y = uint32_t(first / wx % wy), z = uint32_t(first / wx / wy);
    const uint32_t sx = uint32_t(stride % wx), sy = uint32_t(stride / wx % wy), sz = uint32_t(stride / wx / wy);
    for (uint64_t k = first; k < nint; k += stride) {
        const uint64_t i = (x + 1) + uint64_t(p.nx) * ((y + 1) + uint64_t(p.ny) * (z + 1));
        acc.add(macro[M_RHO * N + i], macro[M_UX * N + i], macro[M_UY * N + i], macro[M_UZ * N + i],
                macro[M_PHI * N + i]);
        x += sx;
        y += sy;
        z += sz;
        if (x >= wx) x -= wx, ++y;
        if (y >= wy) y -= wy, ++z;
    }
    double row[RED_FIELDS];
    acc.row(row);
    block_reduce_row<RED_THREADS>(row, partial + size_t(blockIdx.x) * RED_FIELDS);
}

static __global__ void __launch_bounds__(RED_FINAL_THREADS) k_reduce_final(const double *partial, int nblocks,
                                                                           double *out) {
    const int f = threadIdx.x >> 5;
    const double s = red_total(partial, nblocks, f);
    if ((threadIdx.x & 31) == 0) out[f] = s;
}

}  // namespace pflbm

// lattice_f64.cuh - the per-node arithmetic of FP64 runs.
//
// The same algebra as lattice.cuh and stencil.cuh, arranged for the fewest
// FP64 instructions: the unit has 2 lanes per clock and SM, and an FP64 step
// keeps it busy 81% of the time with DRAM at 7% and issue at 8%, so its time
// is the count of FP64 instructions per node. What is shared:
//   - the differences of opposite face diagonals serve two gradient axes
//     (sum and difference), the divergence of the normals takes one weighted
//     sum instead of three, and the factor 3 sits in the weights;
//   - moments: sums and differences of a plane's two diagonals serve the
//     second moments, the density and two momenta; rho u = j + F/2 is formed
//     before the division;
//   - collision: the even part of every direction is w (K + 4.5 c.T.c) with
//     one tensor T = rho u u + sym(u F) + (1 - omega) Pi, the odd part of
//     D3Q19 is 3 w c.(rho u + F/2).
// Every operation but those of the third-order odd part of D3Q27 (make_ctx,
// cdot, hermite3) is rounded by itself (op_*); the plain-load and TMA-fed
// kernels agree bit for bit. D3Q19 jet 96x96x256: 375 -> 284 FP64 instructions
// per interior node (the halo's normals included), 1835 -> 1340 us per collide;
// fields within 4e-14 of the direct forms.
#pragma once
#include "lattice.cuh"
#include "stencil.cuh"

namespace pflbm {

// grad v with the lattice weights (src/phaseField.cuh:67-118), factor 3
// included: v(dx, dy, dz) is a neighbour's value.
template <int QQ, class Get>
__device__ __forceinline__ void gradient_f64(const Get &v, double &gx, double &gy, double &gz) {
    auto sub = [](double a, double b) { return op_add(a, -b); };
    auto pair = [&](int x, int y, int z) { return sub(v(x, y, z), v(-x, -y, -z)); };
    constexpr double w1 = 3.0 * Weights<QQ>::w1, w2 = 3.0 * Weights<QQ>::w2, w3 = 3.0 * Weights<QQ>::w3;
    const double xy = pair(1, 1, 0), xy_ = pair(1, -1, 0), xz = pair(1, 0, 1), xz_ = pair(1, 0, -1),
                 yz = pair(0, 1, 1), yz_ = pair(0, 1, -1);
    gx = op_fma(w1, pair(1, 0, 0), op_mul(w2, op_add(op_add(xy, xy_), op_add(xz, xz_))));
    gy = op_fma(w1, pair(0, 1, 0), op_mul(w2, op_add(sub(xy, xy_), op_add(yz, yz_))));
    gz = op_fma(w1, pair(0, 0, 1), op_mul(w2, op_add(sub(xz, xz_), sub(yz, yz_))));
    if constexpr (QQ == 27) {
        const double a = pair(1, 1, 1), b = pair(1, 1, -1), c = pair(1, -1, 1), d = pair(-1, 1, 1);
        const double ab = op_add(a, b), cd = sub(c, d);
        gx = op_fma(w3, op_add(ab, cd), gx);
        gy = op_fma(w3, sub(ab, cd), gy);
        gz = op_fma(w3, op_add(sub(a, b), op_add(c, d)), gz);
    }
}

// n^ and |grad phi| from the gradient.
__device__ __forceinline__ void unit_normal_f64(double gx, double gy, double gz, double &nx, double &ny, double &nz,
                                                double &ind) {
    ind = sqrt(op_fma(gx, gx, op_fma(gy, gy, op_mul(gz, gz))));
    const double inv = 1.0 / op_add(ind, 1e-9);
    nx = op_mul(gx, inv);
    ny = op_mul(gy, inv);
    nz = op_mul(gz, inv);
}

// div n with the lattice weights, factor 3 included (src/phaseField.cuh:152-212):
// n(c, dx, dy, dz) is component c at a neighbour.
template <int QQ, class Get>
__device__ __forceinline__ double divergence_f64(const Get &n) {
    auto sub = [](double a, double b) { return op_add(a, -b); };
    // (n_a + s n_b) along (1, s), minus the same at the opposite node
    auto diag = [&](int a, int b, int s) {
        int p[3] = {0, 0, 0};
        p[a] = 1;
        p[b] = s;
        const double f = sub(n(a, p[0], p[1], p[2]), n(a, -p[0], -p[1], -p[2]));
        const double g = sub(n(b, p[0], p[1], p[2]), n(b, -p[0], -p[1], -p[2]));
        return s > 0 ? op_add(f, g) : sub(f, g);
    };
    constexpr double w1 = 3.0 * Weights<QQ>::w1, w2 = 3.0 * Weights<QQ>::w2, w3 = 3.0 * Weights<QQ>::w3;
    const double axis = op_add(op_add(sub(n(0, 1, 0, 0), n(0, -1, 0, 0)), sub(n(1, 0, 1, 0), n(1, 0, -1, 0))),
                               sub(n(2, 0, 0, 1), n(2, 0, 0, -1)));
    const double face = op_add(op_add(op_add(diag(0, 1, 1), diag(0, 1, -1)), op_add(diag(0, 2, 1), diag(0, 2, -1))),
                               op_add(diag(1, 2, 1), diag(1, 2, -1)));
    double r = op_fma(w1, axis, op_mul(w2, face));
    if constexpr (QQ == 27) {
        auto body = [&](int x, int y, int z) {
            auto c = [&](int k, int s) {
                const double f = sub(n(k, x, y, z), n(k, -x, -y, -z));
                return s > 0 ? f : -f;
            };
            return op_add(op_add(c(0, x), c(1, y)), c(2, z));
        };
        r = op_fma(w3, op_add(op_add(body(1, 1, 1), body(1, 1, -1)), op_add(body(1, -1, 1), body(-1, 1, 1))), r);
    }
    return r;
}

// moments<QQ, double> (src/lbm.cu:33-128).
template <int QQ>
__device__ __forceinline__ Macro<double> moments_f64(const double (&f)[QQ], double fx, double fy, double fz) {
    constexpr int NP = (QQ - 1) / 2;
    auto sub = [](double a, double b) { return op_add(a, -b); };
    double s[NP], d[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        s[k] = op_add(f[2 * k + 1], f[2 * k + 2]);
        d[k] = sub(f[2 * k + 1], f[2 * k + 2]);
    }
    // pairs: 0-2 the axes, 3 6 / 4 7 / 5 8 the diagonals (1, +-1) of the
    // planes xy, xz, yz
    const double sxy = op_add(s[3], s[6]), sxz = op_add(s[4], s[7]), syz = op_add(s[5], s[8]);
    double mxy = sub(s[3], s[6]), mxz = sub(s[4], s[7]), myz = sub(s[5], s[8]);
    double mxx = op_add(s[0], op_add(sxy, sxz)), myy = op_add(s[1], op_add(sxy, syz)),
           mzz = op_add(s[2], op_add(sxz, syz));
    double r = op_add(op_add(op_add(f[0], mxx), op_add(s[1], s[2])), syz);  // rho - 1
    double jx = op_add(d[0], op_add(op_add(d[3], d[6]), op_add(d[4], d[7])));
    double jy = op_add(d[1], op_add(sub(d[3], d[6]), op_add(d[5], d[8])));
    double jz = op_add(d[2], op_add(sub(d[4], d[7]), sub(d[5], d[8])));
    if constexpr (QQ == 27) {
        const double ab = op_add(s[9], s[10]), cd = op_add(s[11], s[12]), a_b = sub(s[9], s[10]),
                     c_d = sub(s[11], s[12]), all = op_add(ab, cd);
        r = op_add(r, all);
        mxx = op_add(mxx, all);
        myy = op_add(myy, all);
        mzz = op_add(mzz, all);
        mxy = op_add(mxy, sub(ab, cd));
        mxz = op_add(mxz, op_add(a_b, c_d));
        myz = op_add(myz, sub(a_b, c_d));
        const double dab = op_add(d[9], d[10]), dcd = sub(d[11], d[12]);
        jx = op_add(jx, op_add(dab, dcd));
        jy = op_add(jy, sub(dab, dcd));
        jz = op_add(jz, op_add(sub(d[9], d[10]), op_add(d[11], d[12])));
    }
    Macro<double> m;
    m.rho = op_add(r, 1.0);
    const double inv = 1.0 / m.rho;
    const double hx = op_mul(0.5, fx), hy = op_mul(0.5, fy), hz = op_mul(0.5, fz);
    m.ux = op_mul(op_add(jx, hx), inv);
    m.uy = op_mul(op_add(jy, hy), inv);
    m.uz = op_mul(op_add(jz, hz), inv);
    // M_ab - rho u_a u_b + (u_a F_b + u_b F_a) / 2 with rho u = j + F/2
    m.pxx = op_fma(-m.ux, sub(jx, hx), mxx);
    m.pyy = op_fma(-m.uy, sub(jy, hy), myy);
    m.pzz = op_fma(-m.uz, sub(jz, hz), mzz);
    m.pxy = op_fma(m.uy, hx, op_fma(-m.ux, jy, mxy));
    m.pxz = op_fma(m.uz, hx, op_fma(-m.ux, jz, mxz));
    m.pyz = op_fma(m.uz, hy, op_fma(-m.uy, jz, myz));
    const double trace = op_add(op_add(m.pxx, m.pyy), m.pzz);
    m.pxx = op_fma(-1.0 / 3.0, trace, m.pxx);
    m.pyy = op_fma(-1.0 / 3.0, trace, m.pyy);
    m.pzz = op_fma(-1.0 / 3.0, trace, m.pzz);
    return m;
}

// Post-collision shifted populations of every direction (src/lbm.cu:191-206),
// handed to put(q, value).
template <int QQ, class Put>
__device__ __forceinline__ void collide_f64(const Macro<double> &m, double fx, double fy, double fz, double omco,
                                            const Put &put) {
    auto sub = [](double a, double b) { return op_add(a, -b); };
    const double u[3] = {m.ux, m.uy, m.uz}, F[3] = {fx, fy, fz};
    double h[3], k[3], t[3];  // F/2, rho u + F/2, T_aa
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        h[a] = op_mul(0.5, F[a]);
        k[a] = op_fma(m.rho, u[a], h[a]);
        t[a] = op_mul(u[a], op_add(k[a], h[a]));
    }
    const double K = op_fma(-1.5, op_add(op_add(t[0], t[1]), t[2]), op_add(m.rho, -1.0));
    t[0] = op_fma(omco, m.pxx, t[0]);
    t[1] = op_fma(omco, m.pyy, t[1]);
    t[2] = op_fma(omco, m.pzz, t[2]);
    // T_xy, T_xz, T_yz
    const double txy = op_fma(omco, m.pxy, op_fma(u[1], h[0], op_mul(u[0], k[1])));
    const double txz = op_fma(omco, m.pxz, op_fma(u[2], h[0], op_mul(u[0], k[2])));
    const double tyz = op_fma(omco, m.pyz, op_fma(u[2], h[1], op_mul(u[1], k[2])));
    constexpr double w0 = Weights<QQ>::w0, w1 = Weights<QQ>::w1, w2 = Weights<QQ>::w2, w3 = Weights<QQ>::w3;
    put(0, op_mul(w0, K));
    if constexpr (QQ == 19) {
        const double k1 = op_mul(w1, K), k2 = op_mul(w2, K);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double E = op_fma(4.5 * w1, t[a], k1), O = op_mul(3.0 * w1, k[a]);
            put(2 * a + 1, op_add(E, O));
            put(2 * a + 2, sub(E, O));
        }
        const double q[3] = {op_mul(3.0 * w2, k[0]), op_mul(3.0 * w2, k[1]), op_mul(3.0 * w2, k[2])};
        const double off[3] = {op_mul(9.0 * w2, txy), op_mul(9.0 * w2, txz), op_mul(9.0 * w2, tyz)};
        constexpr int A[3] = {0, 0, 1}, B[3] = {1, 2, 2};  // planes xy, xz, yz
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const double e = op_fma(4.5 * w2, op_add(t[A[n]], t[B[n]]), k2);
            const double Ep = op_add(e, off[n]), Em = sub(e, off[n]);
            const double Op = op_add(q[A[n]], q[B[n]]), Om = sub(q[A[n]], q[B[n]]);
            put(7 + 2 * n, op_add(Ep, Op));
            put(8 + 2 * n, sub(Ep, Op));
            put(13 + 2 * n, op_add(Em, Om));
            put(14 + 2 * n, sub(Em, Om));
        }
    } else {
        // odd part with the third-order terms, per pair
        const CollideCtx<double> c = make_ctx<QQ, double>(m, fx, fy, fz, omco);
#pragma unroll
        for (int q = 1; q < QQ; q += 2) {
            const int cx = kCX[q], cy = kCY[q], cz = kCZ[q];
            const int nnz = (cx != 0) + (cy != 0) + (cz != 0);
            const double w = nnz == 1 ? w1 : (nnz == 2 ? w2 : w3);
            double cc = cx != 0 ? t[0] : (cy != 0 ? t[1] : t[2]);  // c.T.c
            if (cx != 0 && cy != 0) cc = op_add(cc, t[1]);
            if ((cx != 0 || cy != 0) && cz != 0) cc = op_add(cc, t[2]);
            if (cx * cy != 0) cc = op_fma(2.0 * (cx * cy), txy, cc);
            if (cx * cz != 0) cc = op_fma(2.0 * (cx * cz), txz, cc);
            if (cy * cz != 0) cc = op_fma(2.0 * (cy * cz), tyz, cc);
            const double E = op_mul(w, op_fma(4.5, cc, K));
            const double cu = cdot<double>(cx, cy, cz, c.u3x, c.u3y, c.u3z), cF = cdot<double>(cx, cy, cz, fx, fy, fz);
            const int cl = weight_class(q);
            const double O = op_fma(op_mul(c.wr[cl], cu), op_fma(op_mul(1.0 / 6.0, cu), cu, c.A),
                                    op_fma(1.5 * w, cF, op_mul(c.ow[cl], hermite3<double>(cx, cy, cz, c))));
            put(q, op_add(E, O));
            put(q + 1, sub(E, O));
        }
    }
}

}  // namespace pflbm

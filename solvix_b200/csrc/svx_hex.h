// svx_hex.h - the C3D8 element operator in registers (device code of
// svx_hex.cu and svx_brick.cu): trilinear modes, gradients at the Gauss points,
// forces.  The arithmetic also compiles for the host, where its test runs.
#ifndef SVX_HEX_H
#define SVX_HEX_H
#ifdef __CUDACC__
#define SVX_HEX_FN __device__ __forceinline__
#else
#define SVX_HEX_FN inline
#endif

namespace svx {

constexpr double HEX_G = 0.57735026918962576450914878050196;  // Gauss abscissa 1 / sqrt(3)

#ifdef __CUDACC__
__device__ __forceinline__ void load_row(const double* p, double (&v)[3]) {
    [[maybe_unused]] double pad;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(pad) : "l"(p));
}
__device__ __forceinline__ void load_row_cg(const double* p, double (&v)[3]) {  // from L2
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
    v[0] = a.x;
    v[1] = a.y;
    v[2] = __ldcg(p + 2);
}
__device__ __forceinline__ void store_row(double* p, double a, double b, double c) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c),
                 "d"(0.0) : "memory");
}

#endif

// Trilinear modes of eight nodal 3-vectors (corner order element.rs:427-437),
// eight times the coefficients of xi, eta, zeta, xi eta, eta zeta, xi zeta
// and xi eta zeta; the products carry their Gauss abscissas (g, g, g, g^2).
struct HexModes {
    double c[7][3];  // one array: the bricks store and load all 21 by one index
    HexModes() = default;
    SVX_HEX_FN double& at(int q) { return c[q / 3][q % 3]; }
    SVX_HEX_FN explicit HexModes(const double (&v)[8][3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            // pairs along xi (0-1, 3-2, 4-5, 7-6), then eta, then zeta
            const double s0 = v[1][k] + v[0][k], d0 = v[1][k] - v[0][k];
            const double s1 = v[2][k] + v[3][k], d1 = v[2][k] - v[3][k];
            const double s2 = v[5][k] + v[4][k], d2 = v[5][k] - v[4][k];
            const double s3 = v[6][k] + v[7][k], d3 = v[6][k] - v[7][k];
            const double ss0 = s1 + s0, sd0 = s1 - s0, ds0 = d1 + d0, dd0 = d1 - d0;
            const double ss1 = s3 + s2, sd1 = s3 - s2, ds1 = d3 + d2, dd1 = d3 - d2;
            c[0][k] = ds1 + ds0;
            c[1][k] = sd1 + sd0;
            c[2][k] = ss1 - ss0;
            c[3][k] = (dd1 + dd0) * HEX_G;
            c[4][k] = (sd1 - sd0) * HEX_G;
            c[5][k] = (ds1 - ds0) * HEX_G;
            c[6][k] = (dd1 - dd0) * (1.0 / 3.0);
        }
    }
    // G[a][k] = eight times d v_k / d xi_a at Gauss point g (bit 2: xi, 1:
    // eta, 0: zeta positive)
    SVX_HEX_FN void gradient(int g, double (&G)[3][3]) const {
        const bool x = g & 4, y = g & 2, z = g & 1;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double a = z ? c[0][k] + c[5][k] : c[0][k] - c[5][k];
            const double b = z ? c[3][k] + c[6][k] : c[3][k] - c[6][k];
            const double d = z ? c[1][k] + c[4][k] : c[1][k] - c[4][k];
            const double e = y ? c[2][k] + c[4][k] : c[2][k] - c[4][k];
            const double f = y ? c[5][k] + c[6][k] : c[5][k] - c[6][k];
            G[0][k] = y ? a + b : a - b;
            G[1][k] = x ? d + b : d - b;
            G[2][k] = x ? e + f : e - f;
        }
    }
};

SVX_HEX_FN double hex_det(const double (&J)[3][3]) {
    return J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
           J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
           J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
}

// Lame constants over the transforms' powers of two (8^3).
SVX_HEX_FN void hex_lame(double E, double nu, double& lam, double& mu) {
    lam = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)) * (1.0 / 512.0);
    mu = E / (2.0 * (1.0 + nu)) * (1.0 / 512.0);
}

// Modal forces of an element.
struct HexForces {
    double f1[3], f2[3], f3[3], f4[3], f5[3], f6[3], f7[3];
    // nodal forces from the modes (the transform of HexModes transposed)
    SVX_HEX_FN void nodal(double (&f)[8][3]) const {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double m4 = f4[c] * HEX_G, m5 = f5[c] * HEX_G, m6 = f6[c] * HEX_G,
                         m7 = f7[c] * (1.0 / 3.0);
            // modes with zeta = -1 and +1
            const double ss0 = -f3[c], ss1 = f3[c];
            const double ds0 = f1[c] - m6, ds1 = f1[c] + m6;
            const double sd0 = f2[c] - m5, sd1 = f2[c] + m5;
            const double dd0 = m4 - m7, dd1 = m4 + m7;
            const double s0 = ss0 - sd0, s1 = ss0 + sd0, s2 = ss1 - sd1, s3 = ss1 + sd1;
            const double d0 = ds0 - dd0, d1 = ds0 + dd0, d2 = ds1 - dd1, d3 = ds1 + dd1;
            f[0][c] = s0 - d0;
            f[1][c] = s0 + d0;
            f[2][c] = s1 + d1;
            f[3][c] = s1 - d1;
            f[4][c] = s2 - d2;
            f[5][c] = s2 + d2;
            f[6][c] = s3 + d3;
            f[7][c] = s3 - d3;
        }
    }
    // u . f over the element (U's products carry g and g^2, the forces not)
    SVX_HEX_FN double work(const HexModes& U) const {
        double w = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            w += ((U.c[0][c] * f1[c] + U.c[1][c] * f2[c]) + (U.c[2][c] * f3[c] + U.c[3][c] * f4[c])) +
                 ((U.c[4][c] * f5[c] + U.c[5][c] * f6[c]) + U.c[6][c] * f7[c]);
        return w;
    }
};

// F = the element's modal forces for displacements U: at each Gauss point
// H = G M with M the (signed, element.rs:448-463) cofactors of J, stresses
// of the symmetric part over det J, and their pull-back by M.  lam and mu
// are the Lame constants over 512, rdet(g) one over the determinant of the
// eightfold Jacobian.  Unrolled: what the Gauss points share is formed once
// (a loop over the (eta, zeta) pairs is 2 KB of code instead of 25 and has a
// tenth more operations; it measured 17.0 against 16.4 us an iteration of the
// whole-device form and 101 against 99 of the graph form).
template <class R>
SVX_HEX_FN void hex_integrate(const HexModes& X, const HexModes& U, double lam,
                                              double mu, R rdet, HexForces& F) {
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        // sums over the plane zeta = -+g: of P_xi, P_eta, P_zeta and of their
        // products with the other coordinates' signs
        double a1[3], a2[3], a3[3], a4[3], a5[3], a6[3], a7[3];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int g = (q << 1) | z;  // bit 2: xi, bit 1: eta
            const bool x = g & 4, y = g & 2;
            double J[3][3], G[3][3];
            X.gradient(g, J);
            U.gradient(g, G);
            double M[3][3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const int a1_ = (a + 1) % 3, a2_ = (a + 2) % 3, b1_ = (b + 1) % 3,
                              b2_ = (b + 2) % 3;
                    M[a][b] = ((a + b) & 1) ? J[a1_][b2_] * J[a2_][b1_] - J[a1_][b1_] * J[a2_][b2_]
                                            : J[a1_][b1_] * J[a2_][b2_] - J[a1_][b2_] * J[a2_][b1_];
                }
            const double w = rdet(g), l = lam * w, m = mu * w;
            double H[3][3];  // H[c][b]
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    H[c][b] = G[0][c] * M[0][b] + G[1][c] * M[1][b] + G[2][c] * M[2][b];
            const double tr = l * (H[0][0] + H[1][1] + H[2][2]), m2 = 2.0 * m;
            const double sx = tr + m2 * H[0][0], sy = tr + m2 * H[1][1], sz = tr + m2 * H[2][2];
            const double sxy = m * (H[0][1] + H[1][0]), syz = m * (H[1][2] + H[2][1]),
                         sxz = m * (H[0][2] + H[2][0]);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double t0 = c == 0 ? sx : c == 1 ? sxy : sxz;
                const double t1 = c == 0 ? sxy : c == 1 ? sy : syz;
                const double t2 = c == 0 ? sxz : c == 1 ? syz : sz;
                const double px = t0 * M[0][0] + t1 * M[0][1] + t2 * M[0][2];
                const double py = t0 * M[1][0] + t1 * M[1][1] + t2 * M[1][2];
                const double pz = t0 * M[2][0] + t1 * M[2][1] + t2 * M[2][2];
                if (q == 0) {
                    a1[c] = px;
                    a2[c] = py;
                    a3[c] = pz;
                    a4[c] = -px - py;
                    a5[c] = -pz;
                    a6[c] = -pz;
                    a7[c] = pz;
                } else {
                    a1[c] += px;
                    a2[c] += py;
                    a3[c] += pz;
                    a4[c] += y ? px : -px;
                    a4[c] += x ? py : -py;
                    a5[c] += y ? pz : -pz;
                    a6[c] += x ? pz : -pz;
                    a7[c] += x == y ? pz : -pz;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (z == 0) {
                F.f1[c] = a1[c];
                F.f2[c] = a2[c];
                F.f3[c] = a3[c];
                F.f4[c] = a4[c];
                F.f5[c] = a5[c] - a2[c];
                F.f6[c] = a6[c] - a1[c];
                F.f7[c] = a7[c] - a4[c];
            } else {
                F.f1[c] += a1[c];
                F.f2[c] += a2[c];
                F.f3[c] += a3[c];
                F.f4[c] += a4[c];
                F.f5[c] += a5[c] + a2[c];
                F.f6[c] += a6[c] + a1[c];
                F.f7[c] += a7[c] + a4[c];
            }
        }
    }
}

}  // namespace svx

#endif  // SVX_HEX_H

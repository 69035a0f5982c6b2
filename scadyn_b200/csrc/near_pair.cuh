// The singularity-subtracted integrals of one near-zone tet pair (constant
// basis): integrate_V_V_G and integrate_dV_dV_G (src/precorrection.f90:729-806)
// over singularity_subtraction_int_V_G / _int_S_G
// (src/singularity_subtraction.f90:112-243) and analytical_integration
// (:15-108), for a thread that holds one pair.
//
// What a pair costs is 52 test points (24 in the volume, 28 on the faces),
// each with the analytic integrals over the four faces of the basis tet and 24
// or 28 values of the Green function.  Everything that depends on the basis
// tet alone (normals, edge directions, in-plane edge normals) is laid out once
// per tet (PairGeo).  Per point the four vertex distances and the six edge
// logarithms serve all faces -- an edge traversed the other way has the same
// integral of 1/R -- and the six arc tangents of a face are one: with
// R0^2 = t^2 + w0^2 the edge terms atan(t s+/(R0^2 + |w0| R+)) -
// atan(t s-/(R0^2 + |w0| R-)) add up to the solid angle of the face, taken from
// its vertex vectors (Van Oosterom and Strackee 1983):
//   tan(Omega/2) = |r1 . (r2 x r3)| / (R1 R2 R3 + (r1.r2) R3 + (r1.r3) R2 + (r2.r3) R1),
// where the triple product is |w0| times twice the face's area.
#pragma once
#include "geom.cuh"

constexpr int PG_V = 0, PG_N = 12, PG_SL = 24, PG_LL = 42, PG_ML = 48, PG_A2 = 84, PG_VOL = 88;
constexpr int PG = 89;       // values per tet, odd: lanes over tets fall in distinct banks

// edges (p, q), p < q, of a tet: 01 02 03 12 13 23
SCD_HD constexpr int pg_edge(int p, int q) { return p > q ? pg_edge(q, p) : p == 0 ? q - 1 : p + q; }
// vertex i of face f (tetra_face, src/common.f90:296-322)
SCD_HD constexpr int pg_face(int f, int i) {
    return f == 0 ? i + 1 : f == 1 ? (i == 0 ? 0 : i == 1 ? 3 : 2) : f == 2 ? (i == 2 ? 3 : i) : (i == 0 ? 0 : i == 1 ? 2 : 1);
}
// start and end vertex of edge l of face f, in analytical_integration's order
SCD_HD constexpr int pg_from(int f, int l) { return pg_face(f, l == 0 ? 1 : l == 1 ? 2 : 0); }
SCD_HD constexpr int pg_to(int f, int l) { return pg_face(f, l == 0 ? 2 : l == 1 ? 0 : 1); }

// what a basis tet's integrals share; item = 0..3 a face, 4..9 an edge
SCD_HD void pair_geo(double *g, const double *v12, double vol, int item) {
    const V3 *v = reinterpret_cast<const V3 *>(v12);
    if (item == 0) {
        for (int i = 0; i < 12; ++i) g[PG_V + i] = v12[i];
        g[PG_VOL] = vol;
    }
    if (item < 4) {
        const int f = item;
        const V3 tri[3] = {v[pg_face(f, 0)], v[pg_face(f, 1)], v[pg_face(f, 2)]};
        const V3 n = tri_normal(tri);
        V3 a, b;
        g[PG_A2 + f] = tri_ww1(tri, a, b);
        g[PG_N + 3 * f] = n.x; g[PG_N + 3 * f + 1] = n.y; g[PG_N + 3 * f + 2] = n.z;
        for (int l = 0; l < 3; ++l) {
            const V3 s = vsub(v[pg_to(f, l)], v[pg_from(f, l)]);
            const double ns = sqrt(vdot(s, s));
            const V3 m = vcross(V3{s.x / ns, s.y / ns, s.z / ns}, n);
            double *o = g + PG_ML + 9 * f + 3 * l;
            o[0] = m.x; o[1] = m.y; o[2] = m.z;
        }
    } else {
        const int e = item - 4, p = e < 3 ? 0 : e < 5 ? 1 : 2, q = e < 3 ? e + 1 : e == 3 ? 2 : 3;
        const V3 s = vsub(v[q], v[p]);
        const double ns = sqrt(vdot(s, s));
        g[PG_LL + e] = ns;
        g[PG_SL + 3 * e] = s.x / ns; g[PG_SL + 3 * e + 1] = s.y / ns; g[PG_SL + 3 * e + 2] = s.z / ns;
    }
}

// g, in a way that keeps the compiler from holding what it reads through it
// across loop iterations: the 89 values of a PairGeo do not fit the registers,
// and spilled copies cost more than shared memory
SCD_HD const double *pair_reload(const double *g) {
#ifdef __CUDA_ARCH__
    int zero = 0;
    asm volatile("" : "+r"(zero));
    return g + zero;
#else
    return g;
#endif
}

// d_v = v - r and |d_v| of the basis tet's vertices for a point r
struct PairPoint {
    V3 d[4];
    double R[4];
    SCD_HD void set(const double *geo, V3 r) {
        const double *g = pair_reload(geo);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            d[v] = V3{g[PG_V + 3 * v] - r.x, g[PG_V + 3 * v + 1] - r.y, g[PG_V + 3 * v + 2] - r.z};
            R[v] = sqrt(vdot(d[v], d[v]));
        }
    }
};

// the integrals of 1/R (K1) and R (K2) over the four faces and the signed
// heights h = (face vertex - r) . n
SCD_HD void pair_analytic(const double *geo, const PairPoint &p, double (&K1)[4], double (&K2)[4], double (&h)[4]) {
    const double *g = pair_reload(geo);
    double I[6], J[6], dd[6];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a + 1; b < 4; ++b) {
            const int e = pg_edge(a, b);
            const V3 sl = V3{g[PG_SL + 3 * e], g[PG_SL + 3 * e + 1], g[PG_SL + 3 * e + 2]};
            const double sm = vdot(p.d[a], sl), sp = sm + g[PG_LL + e];
            const bool first = p.R[a] + sm > p.R[b] - sp;
            const double num = first ? p.R[b] + sp : p.R[a] - sm, den = first ? p.R[a] + sm : p.R[b] - sp;
            I[e] = log(fabs(num / den));
            J[e] = sp * p.R[b] - sm * p.R[a];
            dd[e] = vdot(p.d[a], p.d[b]);
        }
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const int a = pg_face(f, 0), b = pg_face(f, 1), c = pg_face(f, 2);
        const V3 n = V3{g[PG_N + 3 * f], g[PG_N + 3 * f + 1], g[PG_N + 3 * f + 2]};
        h[f] = vdot(p.d[a], n);
        const double w = fabs(h[f]), w2 = w * w;
        double t[3], km1 = 0.0, s2 = 0.0;
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            const int u = pg_from(f, l), e = pg_edge(u, pg_to(f, l));
            const double *m = g + PG_ML + 9 * f + 3 * l;
            t[l] = vdot(p.d[u], V3{m[0], m[1], m[2]});
            km1 += t[l] * I[e];
            s2 += t[l] * (0.5 * (J[e] + (t[l] * t[l] + w2) * I[e]));
        }
        if (w > 1.0e-10) {
            const double den = p.R[a] * p.R[b] * p.R[c] + dd[pg_edge(a, b)] * p.R[c] + dd[pg_edge(a, c)] * p.R[b] +
                               dd[pg_edge(b, c)] * p.R[a];
            km1 -= w * (2.0 * atan2(w * g[PG_A2 + f], den));
        }
        K1[f] = km1;
        K2[f] = 1.0 / 3.0 * (w2 * km1 + s2);
    }
}

// sin x and cos x - 1 for x >= 0: up to 3.2 (a near zone's kR) from Taylor
// polynomials of the half angle (remainders below 3e-18), 2 sin cos and
// -2 sin^2, with neither reduction nor selects; the library's sincos beyond
SCD_HD void sin_cosm1(double x, double &s, double &cm1) {
    if (x <= 3.2) {
        const double y = 0.5 * x, z = y * y;
        double ps = 1.0 / 51090942171709440000.0;
        ps = fma(ps, z, -1.0 / 121645100408832000.0);
        ps = fma(ps, z, 1.0 / 355687428096000.0);
        ps = fma(ps, z, -1.0 / 1307674368000.0);
        ps = fma(ps, z, 1.0 / 6227020800.0);
        ps = fma(ps, z, -1.0 / 39916800.0);
        ps = fma(ps, z, 1.0 / 362880.0);
        ps = fma(ps, z, -1.0 / 5040.0);
        ps = fma(ps, z, 1.0 / 120.0);
        ps = fma(ps, z, -1.0 / 6.0);
        const double h = fma(y * z, ps, y);
        double pc = -1.0 / 1124000727777607680000.0;
        pc = fma(pc, z, 1.0 / 2432902008176640000.0);
        pc = fma(pc, z, -1.0 / 6402373705728000.0);
        pc = fma(pc, z, 1.0 / 20922789888000.0);
        pc = fma(pc, z, -1.0 / 87178291200.0);
        pc = fma(pc, z, 1.0 / 479001600.0);
        pc = fma(pc, z, -1.0 / 3628800.0);
        pc = fma(pc, z, 1.0 / 40320.0);
        pc = fma(pc, z, -1.0 / 720.0);
        pc = fma(pc, z, 1.0 / 24.0);
        pc = fma(pc, z, -0.5);
        const double h2 = h + h;
        s = fma(h2 * z, pc, h2);
        cm1 = -h2 * h;
    } else {
        double h, c;
        sincos(0.5 * x, &h, &c);
        s = 2.0 * h * c;
        cm1 = -2.0 * h * h;
    }
}

// acc += w (exp(ikR)/R - 1/R + k^2 R / 2) for the vector dv of length R, taken
// as at least the cut-off below which the reference puts its limit ik (from
// there both agree to rounding)
SCD_HD void add_green(double &re, double &im, V3 dv, double k, double cut2, double w) {
    const double r2 = fmax(vdot(dv, dv), cut2), ri = rsqrt(r2), R = r2 * ri;
    double s, cm1;
    sin_cosm1(k * R, s, cm1);
    re += w * (cm1 * ri + 0.5 * (k * k) * R);
    im += w * (s * ri);
}

// vvg = integrate_V_V_G, dvv(r + 3 c) = integrate_dV_dV_G of test tet T and
// basis tet B, both as PairGeo; Q supplies the quadrature rules.  acc: 18
// values `stride` apart that hold dvv between the test faces (off the
// registers: it is touched four times).
template <typename Q>
SCD_HD void pair_integrals(const double *T, const double *B, double k, cd &vvg, cd (&dvv)[9], double *acc, int stride) {
    const double c4 = 1.0 / (4 * PI), kk = k * k * (-0.5);
    double K1[4], K2[4], h[4], re = 0.0, im = 0.0;
    {
        const double c = 1.0e-10 * pow(B[PG_VOL], F13_D), cut2 = c * c;
#pragma unroll 1
        for (int i = 0; i < 24; ++i) {
            const double q2 = Q::t5(i, 0), q3 = Q::t5(i, 1), q4 = Q::t5(i, 2), q1 = 1 - q2 - q3 - q4;
            const V3 *tv = reinterpret_cast<const V3 *>(pair_reload(T));
            PairPoint p;
            p.set(B, V3{tv[0].x * q1 + tv[1].x * q2 + tv[2].x * q3 + tv[3].x * q4,
                        tv[0].y * q1 + tv[1].y * q2 + tv[2].y * q3 + tv[3].y * q4,
                        tv[0].z * q1 + tv[1].z * q2 + tv[2].z * q3 + tv[3].z * q4});
            pair_analytic(B, p, K1, K2, h);
            double an = 0.0, gr = 0.0, gi = 0.0;
#pragma unroll
            for (int f = 0; f < 4; ++f) an += h[f] * (K1[f] * 0.5 + kk * (K2[f] * 0.25));
#pragma unroll 1
            for (int j = 0; j < 24; ++j) {
                const double b2 = Q::t5(j, 0), b3 = Q::t5(j, 1), b4 = Q::t5(j, 2), b1 = 1 - b2 - b3 - b4;
                add_green(gr, gi,
                          V3{p.d[0].x * b1 + p.d[1].x * b2 + p.d[2].x * b3 + p.d[3].x * b4,
                             p.d[0].y * b1 + p.d[1].y * b2 + p.d[2].y * b3 + p.d[3].y * b4,
                             p.d[0].z * b1 + p.d[1].z * b2 + p.d[2].z * b3 + p.d[3].z * b4},
                          k, cut2, Q::t5(j, 3));
            }
            const double w = Q::t5(i, 3);
            re += w * (6.0 * B[PG_VOL] * gr + an);
            im += w * (6.0 * B[PG_VOL] * gi);
        }
        vvg = cmk(6.0 * T[PG_VOL] * c4 * re, 6.0 * T[PG_VOL] * c4 * im);
    }
    for (int q = 0; q < 18; ++q) acc[q * stride] = 0.0;
#pragma unroll 1
    for (int ft = 0; ft < 4; ++ft) {
        double ar[4] = {0, 0, 0, 0}, ai[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int i = 0; i < 7; ++i) {
            const double x = Q::r5(i, 0), y = Q::r5(i, 1), w = Q::r5(i, 2);
            const V3 *tv = reinterpret_cast<const V3 *>(pair_reload(T));
            const V3 t0 = tv[face_vertex(ft, 0)], ta = vsub(tv[face_vertex(ft, 1)], t0), tb = vsub(tv[face_vertex(ft, 2)], t0);
            PairPoint p;
            p.set(B, V3{t0.x + ta.x * x + tb.x * y, t0.y + ta.y * x + tb.y * y, t0.z + ta.z * x + tb.z * y});
            pair_analytic(B, p, K1, K2, h);
#pragma unroll
            for (int f = 0; f < 4; ++f) ar[f] += w * (K1[f] + kk * K2[f]);
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                // the seven weights add up to the face's area, half of A2
                const double cut2 = 1.0e-20 * (0.5 * B[PG_A2 + f]);
                const V3 a = p.d[pg_face(f, 0)], b = p.d[pg_face(f, 1)], c = p.d[pg_face(f, 2)];
                double gr = 0.0, gi = 0.0;
#pragma unroll 1
                for (int j = 0; j < 7; ++j) {
                    const double u = Q::r5(j, 0), v = Q::r5(j, 1), o = 1 - u - v;
                    add_green(gr, gi, V3{a.x * o + b.x * u + c.x * v, a.y * o + b.y * u + c.y * v, a.z * o + b.z * u + c.z * v}, k,
                              cut2, Q::r5(j, 2));
                }
                ar[f] += w * B[PG_A2 + f] * gr;
                ai[f] += w * B[PG_A2 + f] * gi;
            }
        }
        const double *tn = T + PG_N + 3 * ft, s = T[PG_A2 + ft] * c4;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const double *bn = B + PG_N + 3 * f;
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double m = tn[r] * bn[c] * s;
                    acc[(r + 3 * c) * stride] += m * ar[f];
                    acc[(9 + r + 3 * c) * stride] += m * ai[f];
                }
        }
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) dvv[q] = cmk(acc[q * stride], acc[(9 + q) * stride]);
}

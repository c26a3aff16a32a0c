// nsfv1_tensor.cuh -- FP64 assembly of quadrilaterals and hexahedra for the plain
// Navier-Stokes flag set, with the element's tensor structure and 2^(dim-1) lanes
// per element.
//
// GB300 takes one FP64 instruction of a warp every 64 clocks per SM sub-partition
// (19 clocks per SM with all four busy), so the time of the FP64 assembly is its
// count of FP64 instructions times the warps of the busiest sub-partition. The
// one-thread-per-element kernels (nsfv1_elem.cuh) execute 13.2 k of them per
// hexahedron for defect + Jacobian, and one colour of a 64^3 mesh is 1,024 warps
// on 608 sub-partitions: some run two while others are done after one. Here:
//  * lane l of an element owns the SCVFs at position (pb, pc) = bits of l across
//    each of the dim edge directions, one direction at a time. In the frame of
//    that edge (along a; b, c counted from the near sides) the shapes and local
//    gradients at the integration point are the same for every lane: products of
//    3/4 (near), 1/4 (far) and 1/2 (along a). Values and gradients of a function
//    are sums and differences along a, then two interpolations (24 operations for
//    all four instead of 32), and the corner gradients g_k, g_k.n and g_k.V come
//    from three numbers each (14 operations for the eight corners, not 24);
//  * on affine elements J^-T, the SCVF normals (cofactors of J over 4) and the SCV
//    volume are computed once per lane; elsewhere J and the normal per SCVF;
//  * LPS on affine elements: the upwind exit parameter is the reciprocal of the
//    largest |w_a| / distance, which is |v| / L_up itself (no square root and no
//    cross-multiplied divisions); an exit point lies on a face, so its velocity is
//    a sum over four corners picked from shared memory and the shapes are four
//    products placed by selects;
//  * |v| / L and 1 / L come from one reciprocal square root each;
//  * the Jacobian blocks of a warp pass through shared memory and are reduced into the
//    matrix by consecutive entries.
// Counted per hexahedron: 7.7 k FP64 instructions for LPS + FLOW defect and Jacobian (13.2 k
// before), with the FP64 pipe 77 % active (its practical limit is 16/19). Measured, one thread
// per element before -> here: 64^3 affine, defect + Jacobian 7.73 -> 4.47 ms; 41^3 distorted
// transient, defect 2.56 -> 0.92 ms; 32^2 quadrilaterals 293 -> 118 us (143 without SPLIT). With 8-byte reductions
// straight from the lanes the first was 5.6 ms (138 G sectors/s into L2).
//
// Determinism: the SCVFs of one direction touch disjoint rows, and __syncwarp
// orders the directions, so every address still gets its contributions in a fixed
// order (colours, then directions).
#pragma once
#include "nsfv1_asm_common.cuh"

namespace nsfv1 {

// the calls the tensor and simplex kernels serve (everything else takes the kernels of nsfv1_elem.cuh);
// 'jac': the call forms the Jacobian
inline bool plain_params(const DiscParams& P, const bool jac) {
    return !P.stokes && !P.laplace && !P.peclet && !P.pac && (!jac || P.fullNewton == 0.0) && P.diffLen == DL_RAW &&
           (P.stab == STAB_FIELDS || P.stab == STAB_FLOW) && P.sameUpwind &&
           (P.convUpwind == UPW_NO || P.convUpwind == UPW_FULL || P.convUpwind == UPW_LPS);
}

// |v| from v^2 in one reciprocal square root; 0, an overflowed square and NaN as the square root has
// them (the range test on the bits: a comparison is an FP64 instruction)
__device__ __forceinline__ double speed(const double vv) {
    return (unsigned long long)(__double_as_longlong(vv) - 1) < 0x7fefffffffffffffULL ? vv * rsqrt(vv) : vv;
}

template <int DIM, bool SPLIT = false>
struct Ten {
    static_assert(DIM == 2 || !SPLIT, "a lane per SCVF for quadrilaterals only");
    static constexpr int NSH = 1 << DIM, L = SPLIT ? NSH : NSH / 2, B = DIM + 1, EPW = 32 / L;
    static constexpr int CPL = NSH / L;   // corners that a lane loads
    // corner with bits (x, y, z) in the reference element's order
    static __device__ __forceinline__ int corner(const int bits) {
        const int x = bits & 1, y = (bits >> 1) & 1;
        return (x ^ y) + 2 * y + (DIM == 3 ? (bits & 4) : 0);
    }
    // shared memory of an element: coordinates, state, old velocity, then the edge vectors and
    // cofactors (affine) or the SCV volumes
    static constexpr int DOUBLES = NSH * (2 * DIM + B) + 2 * DIM * DIM;
    // the warp's blocks on their way to the reductions, one per lane (odd stride: no bank conflicts)
    static constexpr int BB = B * B, STRIDE = BB | 1;
    static constexpr int warp_doubles(const bool jac) { return DOUBLES * EPW + (jac ? 32 * STRIDE : 0); }
};

// value and local gradients at the integration point from the NSH corner values of the edge
// frame (index = along a + 2 (far in b) + 4 (far in c))
template <int DIM>
__device__ __forceinline__ void ten_interp(const double (&U)[1 << DIM], double& val, double (&gl)[DIM]) {
    if constexpr (DIM == 3) {
        const double m0 = U[0] + U[1], m1 = U[2] + U[3], m2 = U[4] + U[5], m3 = U[6] + U[7];
        const double d0 = U[1] - U[0], d1 = U[3] - U[2], d2 = U[5] - U[4], d3 = U[7] - U[6];
        val = fma(9.0, m0, fma(3.0, m1 + m2, m3)) * 0.03125;
        gl[0] = fma(9.0, d0, fma(3.0, d1 + d2, d3)) * 0.0625;
        gl[1] = fma(3.0, m1 - m0, m3 - m2) * 0.125;
        gl[2] = fma(3.0, m2 - m0, m3 - m1) * 0.125;
    } else {
        const double m0 = U[0] + U[1], m1 = U[2] + U[3];
        val = fma(3.0, m0, m1) * 0.125;
        gl[0] = fma(3.0, U[1] - U[0], U[3] - U[2]) * 0.25;
        gl[1] = (m1 - m0) * 0.5;
    }
}

// z . grad N_k of the two corners k of edge q of the edge frame (q = far in b + 2 (far in c))
// from t_c = (column c of J^-T) . z
template <int DIM>
__device__ __forceinline__ void ten_pattern(const int q, const double (&t)[DIM], double& lo, double& hi) {
    double x, y;
    if constexpr (DIM == 3) {
        const int c = DIM - 1;
        x = q == 0 ? 0.5625 : q == 3 ? 0.0625 : 0.1875;
        y = q == 0 ? fma(-0.375, t[1], -0.375 * t[c]) : q == 1 ? fma(0.375, t[1], -0.125 * t[c])
          : q == 2 ? fma(-0.125, t[1], 0.375 * t[c]) : fma(0.125, t[1], 0.125 * t[c]);
    } else {
        x = q == 0 ? 0.75 : 0.25;
        y = q == 0 ? -0.5 * t[1] : 0.5 * t[1];
    }
    lo = fma(-x, t[0], y);
    hi = fma(x, t[0], y);
}

template <int DIM> __device__ __forceinline__ double ten_shape(const int r) {
    const int far = DIM == 3 ? ((r >> 1) & 1) + ((r >> 2) & 1) : (r >> 1) & 1;
    if (DIM == 3) return far == 0 ? 0.28125 : far == 1 ? 0.09375 : 0.03125;
    return far == 0 ? 0.375 : 0.125;
}

// SCV volume of one corner of a hexahedron: the six tetrahedra around the diagonal corner -
// centre share it, so their sum is one dot product of it with three cross products
// (D: the other corners relative to this one, index = bits of the directions crossed)
__device__ __forceinline__ double hex_scv(const double (&D)[8][3]) {
    double f01[3], f02[3], f12[3], c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        f01[d] = D[1][d] + D[2][d] + D[3][d];
        f02[d] = D[1][d] + D[4][d] + D[5][d];
        f12[d] = D[2][d] + D[4][d] + D[6][d];
        c[d] = f01[d] + (D[4][d] + D[5][d]) + (D[6][d] + D[7][d]);
    }
    double s[3] = {0.0, 0.0, 0.0};
    auto cross = [&](const double (&f)[3], const double (&p)[3], const double (&q)[3]) {
        const double e0 = p[0] - q[0], e1 = p[1] - q[1], e2 = p[2] - q[2];
        s[0] = fma(f[1], e2, fma(-f[2], e1, s[0]));
        s[1] = fma(f[2], e0, fma(-f[0], e2, s[1]));
        s[2] = fma(f[0], e1, fma(-f[1], e0, s[2]));
    };
    cross(f01, D[2], D[1]);
    cross(f12, D[4], D[2]);
    cross(f02, D[1], D[4]);
    return fabs(s[0] * c[0] + s[1] * c[1] + s[2] * c[2]) * (1.0 / 384.0);
}

// The velocity at the point of the affine LPS ray on the element's surface, and its shapes.
// t: coordinates of the point (t[e] is 0 or 1), e: the axis it left through, hi: t[e] == 1.
// us(f, r): state of function f at corner r of the edge frame (shared memory).
template <int DIM, bool SHAPES, class US>
__device__ __forceinline__ void ten_exit(const double (&t)[DIM], const int e, const bool hi, const US& us, double (&v)[DIM], double* sh) {
    if constexpr (DIM == 3) {
        // the two other axes, in increasing order
        const double p = e == 0 ? t[1] : t[0], q = e == 2 ? t[1] : t[2];
        const int sp = e == 0 ? 2 : 1, sq = e == 2 ? 2 : 4, base = hi ? 1 << e : 0;
        const double p1 = 1.0 - p, q1 = 1.0 - q;
        const double w[4] = {p1 * q1, p * q1, p1 * q, p * q};
#pragma unroll
        for (int d = 0; d < 3; ++d)
            v[d] = fma(w[3], us(d, base + sp + sq), fma(w[2], us(d, base + sq), fma(w[1], us(d, base + sp), w[0] * us(d, base))));
        if constexpr (SHAPES) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int ba = r & 1, bb = (r >> 1) & 1, bc = r >> 2;
                const bool on = (((r >> e) & 1) != 0) == hi;
                const double s0 = w[bb + 2 * bc], s1 = w[ba + 2 * bc], s2 = w[ba + 2 * bb];
                const double s = e == 0 ? s0 : e == 1 ? s1 : s2;
                sh[r] = on ? s : 0.0;
            }
        }
    } else {
        const double p = e == 0 ? t[1] : t[0], p1 = 1.0 - p;
        const int sp = e == 0 ? 2 : 1, base = hi ? 1 << e : 0;
#pragma unroll
        for (int d = 0; d < 2; ++d) v[d] = fma(p, us(d, base + sp), p1 * us(d, base));
        if constexpr (SHAPES) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const bool on = (((r >> e) & 1) != 0) == hi;
                const bool far = e == 0 ? (r >> 1) : (r & 1);
                sh[r] = on ? (far ? p : p1) : 0.0;
            }
        }
    }
}

// One colour's elements [0, count) of A.elems, all affine or (AFFINE = false) any; LPS only
// with AFFINE. JAC: the Jacobian, and the defect if A.D is set; else the defect alone.
// FLOW: the FLOW stabilisation, else FIELDS.
// SPLIT (quadrilaterals): a lane per SCVF instead of one per position with both directions, for
// launches of few warps, whose time is a lane's serial chain. Lanes of the two directions meet
// in the same rows; their reductions take turns.
// Registers: the 3D Jacobian gets two CTAs a SM (254 registers, no spills): bounded to three (168) the 64^3
// pass took 4.64 ms instead of 4.47. The others fit three without spills.
template <int DIM, bool JAC, bool FLOW, bool AFFINE, bool SPLIT = false>
__global__ void __launch_bounds__(kThreads, DIM == 3 && JAC ? 2 : 3) k_tensor(const DiscParams P, const AsmArgs A) {
    using T = Ten<DIM, SPLIT>;
    constexpr int NSH = T::NSH, L = T::L, B = T::B, EPW = T::EPW, Pc = DIM, CPL = T::CPL;
    extern __shared__ double smem[];
    const bool tr = P.transient != 0, def = !JAC || A.D != nullptr;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = lane / L, l = lane - grp * L;
    const int64_t t = ((int64_t)blockIdx.x * (blockDim.x >> 5) + warp) * EPW + grp;
    // lanes without an element (past the end, inactive instance) follow the warp on a valid one and
    // add nothing: the reductions below are formed by all lanes together
    bool valid = t < A.count;
    const int32_t e = __ldg(A.elems + (valid ? t : (int64_t)A.count - 1));
    if (A.elemInst && !__ldg(A.instActive + __ldg(A.elemInst + e))) valid = false;
    if (!__any_sync(0xffffffffu, valid)) return;
    const int32_t* __restrict__ conn = A.conn + (int64_t)e * NSH;
    double* sx = smem + (size_t)warp * T::warp_doubles(JAC) + grp;             // [DIM][NSH][EPW]
    double* su = sx + DIM * NSH * EPW;                                          // [B][NSH][EPW]
    double* so = su + B * NSH * EPW;                                            // [DIM][NSH][EPW] (implicit Euler)
    double* sv = so + DIM * NSH * EPW;                                          // [NSH][EPW] SCV volumes (general elements)
    auto sE = [&](const int c, const int d) -> double& { return sv[(c * DIM + d) * EPW]; };                    // edge vectors (affine)
    auto sC = [&](const int c, const int d) -> double& { return sv[(DIM * DIM + c * DIM + d) * EPW]; };        // cofactors (affine)
    // ---- gather: this lane's corners (the ends of its edge along x; one corner with SPLIT)
    const int l0 = CPL * l;                    // bits (x, y, z) of the first
    const int c0 = T::corner(l0), c1 = T::corner(l0 + CPL - 1);
    int32_t nd0 = __ldg(conn + c0), nd1 = __ldg(conn + c1);
#ifdef NSFV1_BOUNDS_CHECK
    {
        const bool in = NSFV1_IN_RANGE(nd0, A.nNodes, A.err) && NSFV1_IN_RANGE(nd1, A.nNodes, A.err);
        const unsigned group = ((1u << L) - 1u) << (grp * L);   // the lanes of this element
        if ((__ballot_sync(0xffffffffu, in) & group) != group) valid = false;
        if (!in) nd0 = nd1 = 0;
    }
#endif
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        sx[(d * NSH + l0) * EPW] = __ldg(A.coords + (int64_t)nd0 * DIM + d);
        if (CPL == 2) sx[(d * NSH + l0 + 1) * EPW] = __ldg(A.coords + (int64_t)nd1 * DIM + d);
        if (tr && def) {
            so[(d * NSH + l0) * EPW] = __ldg(A.Uold + (int64_t)nd0 * B + d);
            if (CPL == 2) so[(d * NSH + l0 + 1) * EPW] = __ldg(A.Uold + (int64_t)nd1 * B + d);
        }
    }
#pragma unroll
    for (int f = 0; f < B; ++f) {
        su[(f * NSH + l0) * EPW] = __ldg(A.U + (int64_t)nd0 * B + f);
        if (CPL == 2) su[(f * NSH + l0 + 1) * EPW] = __ldg(A.U + (int64_t)nd1 * B + f);
    }
    __syncwarp();
    const double nu = A.nuElem ? __ldg(A.nuElem + e) : P.nu;
    const double rho = P.rho, mnr = -1.0 * nu * rho;
    double irho = 1.0, idt = 0.0;
    if (rho != 1.0) irho = 1.0 / rho;
    if (tr) idt = 1.0 / P.dt;
    const double js = tr ? P.dt : 1.0;
    const int upw = P.convUpwind;
    const int pb = l & 1, pc = DIM == 3 ? l >> 1 : 0, ax = SPLIT ? l >> 1 : 0;
    bool ok = true;
    double* sblk = smem + (size_t)warp * T::warp_doubles(JAC) + T::DOUBLES * EPW;   // [32][STRIDE] (JAC)

    // ---- element geometry. Affine: edge vectors E_c along the axes, cofactors C_c (the SCVF normal
    // of axis c is C_c / 2^(DIM-1), column c of J^-T is C_c / det); lane c forms those of axis c
    double id = 0.0, vol = 0.0;
    if constexpr (AFFINE) {
        if (l < DIM)
#pragma unroll
            for (int d = 0; d < DIM; ++d) sE(l, d) = sx[(d * NSH + (1 << l)) * EPW] - sx[(d * NSH) * EPW];
        __syncwarp();
        if (l < DIM) {
            if constexpr (DIM == 3) {
                const int p = l == 2 ? 0 : l + 1, q = l == 0 ? 2 : l - 1;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int d1 = (d + 1) % 3, d2 = (d + 2) % 3;
                    sC(l, d) = sE(p, d1) * sE(q, d2) - sE(p, d2) * sE(q, d1);
                }
            } else {
                sC(l, 0) = l ? flip_sign(sE(0, 1)) : sE(1, 1);
                sC(l, 1) = l ? sE(0, 0) : flip_sign(sE(1, 0));
            }
        }
        __syncwarp();
        double det = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) det = fma(sE(0, d), sC(0, d), det);
        vol = fabs(det) * (DIM == 3 ? 0.125 : 0.25);
        id = 1.0 / det;
    } else {
        // SCV volumes of this lane's two corners
        if constexpr (DIM == 3) {
#pragma unroll 1
            for (int k = 0; k < 2; ++k) {
                double D[8][3];
#pragma unroll
                for (int q = 0; q < 8; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) D[q][d] = q ? sx[(d * NSH + ((l0 + k) ^ q)) * EPW] - sx[(d * NSH + l0 + k) * EPW] : 0.0;
                sv[(l0 + k) * EPW] = hex_scv(D);
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < CPL; ++k) {
                // corner - edge midpoint - centre - edge midpoint: half the cross product of the
                // diagonals (centre - corner) and (midpoint - midpoint)
                double x0[2], x1[2], x2[2], x3[2];
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    x0[d] = sx[(d * NSH + l0 + k) * EPW];
                    x1[d] = sx[(d * NSH + ((l0 + k) ^ 1)) * EPW] - x0[d];
                    x2[d] = sx[(d * NSH + ((l0 + k) ^ 2)) * EPW] - x0[d];
                    x3[d] = sx[(d * NSH + ((l0 + k) ^ 3)) * EPW] - x0[d];
                }
                const double s0 = x1[0] + x2[0] + x3[0], s1 = x1[1] + x2[1] + x3[1];
                sv[(l0 + k) * EPW] = fabs(s0 * (x2[1] - x1[1]) - s1 * (x2[0] - x1[0])) * 0.0625;
            }
        }
        __syncwarp();
    }

    // ---- one SCVF per axis a; b, c the next axes in cyclic order
#pragma unroll 1
    for (int a = ax; a < (SPLIT ? ax + 1 : DIM); ++a) {
        const int sa = 1 << a, sb = 1 << (DIM == 3 ? (a + 1) % 3 : 1 - a), sc = DIM == 3 ? 1 << ((a + 2) % 3) : 0;
        // bits of corner r of the edge frame
        const int near = (pb ? sb : 0) + (pc ? sc : 0);
        auto bits = [&](const int r) { return near ^ ((r & 1 ? sa : 0) + (r & 2 ? sb : 0) + (r & 4 ? sc : 0)); };
        auto us = [&](const int f, const int r) { return su[(f * NSH + bits(r)) * EPW]; };
        // orientation of the reference element's edge (it decides the upwind corner of a zero flux)
        const bool plus = a == 0 ? !(near & 2) : a == 1 ? (near & 1) != 0 : true;

        const int32_t clow = T::corner(near), chigh = T::corner(near ^ sa);
        // the block indices of this SCVF's two rows, requested long before their use
        int32_t ql[JAC ? NSH : 1], qh[JAC ? NSH : 1];
        if constexpr (JAC) {
            const int32_t* __restrict__ bl = A.elemBlk + (int64_t)e * NSH * NSH;
#pragma unroll
            for (int r = 0; r < NSH; ++r) {
                const int k = T::corner(bits(r));
                ql[r] = __ldg(bl + clow * NSH + k);
                qh[r] = __ldg(bl + chigh * NSH + k);
                if (!valid || !NSFV1_IN_RANGE(ql[r], A.nnzb, A.err)) ql[r] = -1;
                if (!valid || !NSFV1_IN_RANGE(qh[r], A.nnzb, A.err)) qh[r] = -1;
            }
        }
        // values and local gradients of every function
        double val[B], gl[B][DIM], u0[DIM], u1[DIM];
#pragma unroll
        for (int f = 0; f < B; ++f) {
            double U[NSH];
#pragma unroll
            for (int r = 0; r < NSH; ++r) U[r] = us(f, r);
            ten_interp<DIM>(U, val[f], gl[f]);
            if (f < DIM) { u0[f] = U[0]; u1[f] = U[1]; }
        }
        // geometry of the SCVF: normal n (along +a), J^-T columns Gp of the edge frame
        double n[DIM], Gp[DIM][DIM], area, ds = 0.0, lowL2 = 0.0, highL2 = 0.0;
        if constexpr (AFFINE) {
            const double h = DIM == 3 ? 0.25 : 0.5;
            const int ab = DIM == 3 ? (a == 2 ? 0 : a + 1) : 1 - a, ac = a == 0 ? 2 : a - 1;
            double E0[DIM], Eb[DIM], Ec[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double c0 = sC(a, d);
                n[d] = h * c0;
                Gp[0][d] = c0 * id;
                const double gb = sC(ab, d) * id;
                Gp[1][d] = pb ? flip_sign(gb) : gb;
                E0[d] = sE(a, d);
                Eb[d] = sE(ab, d);
                if constexpr (DIM == 3) {
                    const double gc = sC(ac, d) * id;
                    Gp[DIM - 1][d] = pc ? flip_sign(gc) : gc;
                    Ec[d] = sE(ac, d);
                }
            }
            area = vol * vol;
            // z = edge midpoint -> centre; the integration point is half way
            double z[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double zb = pb ? flip_sign(Eb[d]) : Eb[d];
                if constexpr (DIM == 3) z[d] = 0.5 * (zb + (pc ? flip_sign(Ec[d]) : Ec[d]));
                else z[d] = 0.5 * zb;
            }
            if constexpr (DIM == 3) ds = z[0] * z[0] + z[1] * z[1] + z[2] * z[2];
            if (upw == UPW_FULL) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double lo = 0.5 * (z[d] + E0[d]), hi = 0.5 * (z[d] - E0[d]);
                    lowL2 = fma(lo, lo, lowL2);
                    highL2 = fma(hi, hi, highL2);
                }
            }
        } else {
            double J[DIM][DIM], z[DIM], w[DIM], xl[DIM], xh[DIM], gip[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                double X[NSH], v, g[DIM];
#pragma unroll
                for (int r = 0; r < NSH; ++r) X[r] = sx[(d * NSH + bits(r)) * EPW];
                ten_interp<DIM>(X, v, g);
#pragma unroll
                for (int c = 0; c < DIM; ++c) J[d][c] = g[c];
                xl[d] = X[0]; xh[d] = X[1];
                const double m0 = X[0] + X[1], m1 = X[2] + X[3], em = 0.5 * m0;
                if constexpr (DIM == 3) {
                    const double m2 = X[4] + X[5], m3 = X[6] + X[7];
                    const double fb = 0.25 * (m0 + m2), fc = 0.25 * (m0 + m1), ce = 0.125 * ((m0 + m1) + (m2 + m3));
                    z[d] = ce - em;
                    w[d] = fb - fc;
                    gip[d] = 0.25 * ((em + ce) + (fb + fc));
                } else {
                    const double ce = 0.25 * (m0 + m1);
                    z[d] = ce - em;
                    gip[d] = 0.5 * (em + ce);
                }
            }
            if constexpr (DIM == 3) {
                const double h = pb ^ pc ? -0.5 : 0.5;
                n[0] = h * (z[1] * w[2] - z[2] * w[1]);
                n[1] = h * (z[2] * w[0] - z[0] * w[2]);
                n[2] = h * (z[0] * w[1] - z[1] * w[0]);
                ds = z[0] * z[0] + z[1] * z[1] + z[2] * z[2];
                double C[3][3];
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const int c1i = (c + 1) % 3, c2i = (c + 2) % 3, d1 = (d + 1) % 3, d2 = (d + 2) % 3;
                        C[c][d] = J[d1][c1i] * J[d2][c2i] - J[d2][c1i] * J[d1][c2i];
                    }
                const double idet = 1.0 / (J[0][0] * C[0][0] + J[1][0] * C[0][1] + J[2][0] * C[0][2]);
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int d = 0; d < 3; ++d) Gp[c][d] = C[c][d] * idet;
            } else {
                const bool flip = (pb ^ a) != 0;
                n[0] = flip ? -z[1] : z[1];
                n[1] = flip ? z[0] : -z[0];
                const double idet = 1.0 / (J[0][0] * J[1][1] - J[0][1] * J[1][0]);
                Gp[0][0] = J[1][1] * idet; Gp[0][1] = -J[0][1] * idet;
                Gp[1][0] = -J[1][0] * idet; Gp[1][1] = J[0][0] * idet;
            }
            area = 0.5 * (sv[near * EPW] + sv[(near ^ sa) * EPW]);
            area *= area;
            if (upw == UPW_FULL) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double lo = gip[d] - xl[d], hi = gip[d] - xh[d];
                    lowL2 = fma(lo, lo, lowL2);
                    highL2 = fma(hi, hi, highL2);
                }
            }
        }
        double nn = 0.0, vv = 0.0, Vn = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            nn = fma(n[d], n[d], nn);
            vv = fma(val[d], val[d], vv);
            Vn = fma(n[d], val[d], Vn);
        }
        if constexpr (DIM == 2) ds = nn;
        const double nuL = nu * (nn / (0.5 * area + 0.375 * ds * nn));
        // reference-coordinate velocity w = J^-1 v of the edge frame (FLOW, LPS)
        double w[DIM];
#pragma unroll
        for (int c = 0; c < DIM; ++c) w[c] = 0.0;
        if (FLOW || upw == UPW_LPS) {
#pragma unroll
            for (int c = 0; c < DIM; ++c)
#pragma unroll
                for (int d = 0; d < DIM; ++d) w[c] = fma(Gp[c][d], val[d], w[c]);
        }
        // ---- upwind (and downwind) velocity, shapes and coefficients: ncl = |v| / L_up,
        // ndl = |v| / (L_down + L_up)
        double upv[DIM], dnv[DIM], up[NSH], dn[NSH], ncl, ndl = 0.0;
        const double norm = (upw != UPW_LPS || vv < 1.01e-28) ? speed(vv) : 1.0;
        if (upw == UPW_FULL) {
            const bool low = plus ? Vn > 0.0 : !(Vn < 0.0);
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                upv[d] = low ? u0[d] : u1[d];
                dnv[d] = low ? u1[d] : u0[d];
            }
#pragma unroll
            for (int r = 0; r < NSH; ++r) {
                up[r] = r == 0 ? (low ? 1.0 : 0.0) : r == 1 ? (low ? 0.0 : 1.0) : 0.0;
                dn[r] = r == 0 ? (low ? 0.0 : 1.0) : r == 1 ? (low ? 1.0 : 0.0) : 0.0;
            }
            // the downwind corner of -v: the same tie rule on the negated flux
            if (Vn == 0.0) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) dnv[d] = upv[d];
                dn[0] = up[0]; dn[1] = up[1];
            }
            const double ru = rsqrt(low ? lowL2 : highL2);
            ncl = norm * ru;
            if constexpr (FLOW) {
                const double l2 = Vn == 0.0 ? (low ? lowL2 : highL2) : (low ? highL2 : lowL2);
                const double Lu = (low ? lowL2 : highL2) * ru, Ld = l2 * rsqrt(l2);
                ndl = norm / (Ld + Lu);
            }
        } else if (upw == UPW_LPS && AFFINE && !(norm < 1e-14)) {
            // distance to the near side 1/4, to the far side 3/4 (1/2 along a): the ray along -w
            // leaves through the side with the largest |w| / distance
            double bu = 0.0, bd = 0.0;
            int eu = -1, ed = -1;
            bool hu = false, hd = false;
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
                const double aw = fabs(w[c]);
                const bool pos = w[c] > 0.0;
                const double rn = c == 0 ? 2.0 * aw : 4.0 * aw, rf = c == 0 ? rn : aw * (4.0 / 3.0);
                const double ru = pos ? rn : rf, rd = pos ? rf : rn;
                if (ru > bu) { bu = ru; eu = c; hu = !pos; }
                if (FLOW && rd > bd) { bd = rd; ed = c; hd = pos; }
            }
            if (eu < 0) { ok = false; eu = 0; }   // a velocity that is not a number
            ncl = bu;
            const double s = 1.0 / bu;
            double p[DIM];
#pragma unroll
            for (int c = 0; c < DIM; ++c) p[c] = fma(-s, w[c], c == 0 ? 0.5 : 0.25);
            ten_exit<DIM, JAC>(p, eu, hu, us, upv, up);
            if constexpr (FLOW) {
                if (ed < 0) ed = 0;
                const double sd = 1.0 / bd;
                ndl = 1.0 / (s + sd);
#pragma unroll
                for (int c = 0; c < DIM; ++c) p[c] = fma(sd, w[c], c == 0 ? 0.5 : 0.25);
                ten_exit<DIM, JAC>(p, ed, hd, us, dnv, dn);
            }
        } else {
            // no upwind: the interpolation; LPS without a velocity: zero shapes
            const bool zero = upw == UPW_LPS;
#pragma unroll
            for (int d = 0; d < DIM; ++d) upv[d] = dnv[d] = zero ? 0.0 : val[d];
#pragma unroll
            for (int r = 0; r < NSH; ++r) up[r] = dn[r] = zero ? 0.0 : ten_shape<DIM>(r);
            ncl = norm;
            if constexpr (FLOW) ndl = 0.5 * norm;
        }
        double diag = nuL + ncl;
        if (tr) diag += idt;
        const double idiag = 1.0 / diag;
        const double cu = FLOW ? ncl - ndl : ncl;

        if (def) {
            // G^T n and the gradients against the normal: du_d/dn and sum_q n_q du_q/dx_d
            double gn[DIM], q[DIM], trace = 0.0, contN = 0.0, flux[DIM];
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
                gn[c] = 0.0; q[c] = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    gn[c] = fma(Gp[c][d], n[d], gn[c]);
                    q[c] = fma(gl[d][c], n[d], q[c]);
                    if constexpr (FLOW) trace = fma(Gp[c][d], gl[d][c], trace);
                }
            }
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                double s = 0.0, gp = 0.0, cv = 0.0;
#pragma unroll
                for (int c = 0; c < DIM; ++c) {
                    s = fma(gl[d][c], gn[c], s);
                    s = fma(Gp[c][d], q[c], s);
                    gp = fma(Gp[c][d], gl[Pc][c], gp);
                    if constexpr (FLOW) cv = fma(w[c], gl[d][c], cv);
                }
                double rhs = P.hasSource ? P.src[d] : 0.0;
                if (tr) {
                    double O[NSH], ov;
                    double og[DIM];
#pragma unroll
                    for (int r = 0; r < NSH; ++r) O[r] = so[(d * NSH + bits(r)) * EPW];
                    ten_interp<DIM>(O, ov, og);
                    rhs = fma(ov, idt, rhs);
                }
                rhs = fma(nuL, val[d], rhs);
                rhs = fma(cu, upv[d], rhs);
                if constexpr (FLOW) rhs = fma(ndl, dnv[d], rhs) + (val[d] * trace - cv);
                rhs = fma(-irho, gp, rhs);
                contN = fma(rhs * idiag, n[d], contN);
                flux[d] = fma(s, mnr, fma(upv[d], rho * Vn, val[Pc] * n[d]));
            }
            double* __restrict__ dl = A.D + (int64_t)__ldg(conn + clow) * B;
            double* __restrict__ dh = A.D + (int64_t)__ldg(conn + chigh) * B;
            auto reduce = [&]() {
#pragma unroll
                for (int f = 0; f < B; ++f) {
                    double v = f < DIM ? flux[f < DIM ? f : 0] : contN * rho;
                    if (tr) v *= js;
                    atomicAdd(dl + f, v);
                    atomicAdd(dh + f, flip_sign(v));
                }
            };
            if constexpr (SPLIT) {
                if (valid && ax == 0) reduce();
                __syncwarp();
                if (valid && ax == 1) reduce();
                __syncwarp();
            } else {
                if (valid) reduce();
            }
        }
        if constexpr (JAC) {
            double tn[DIM], tv[DIM], mn[DIM], rin[DIM], pn[DIM];
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
                tn[c] = 0.0; tv[c] = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) tn[c] = fma(Gp[c][d], n[d], tn[c]);
                if constexpr (FLOW) tv[c] = w[c];
            }
            const double m = mnr * js, ri = rho * idiag * js, pw = Vn * rho * js, riVn = ri * Vn, ppr = -(idiag * js);
#pragma unroll
            for (int d = 0; d < DIM; ++d) { mn[d] = m * n[d]; rin[d] = ri * n[d]; pn[d] = js * n[d]; }
            double* __restrict__ vals = reinterpret_cast<double*>(A.vals);
#pragma unroll
            for (int q = 0; q < NSH / 2; ++q) {
                double g[2][DIM], gnk[2], vgk[2] = {0.0, 0.0};
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    double td[DIM];
#pragma unroll
                    for (int c = 0; c < DIM; ++c) td[c] = Gp[c][d];
                    ten_pattern<DIM>(q, td, g[0][d], g[1][d]);
                }
                ten_pattern<DIM>(q, tn, gnk[0], gnk[1]);
                if constexpr (FLOW) ten_pattern<DIM>(q, tv, vgk[0], vgk[1]);
                const double N = ten_shape<DIM>(2 * q), nuN = nuL * N;
                double pN[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) pN[d] = N * pn[d];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = 2 * q + h;
                    double Bk[B][B];
                    const double dd = fma(up[r], pw, m * gnk[h]);
#pragma unroll
                    for (int d1 = 0; d1 < DIM; ++d1) {
#pragma unroll
                        for (int d2 = 0; d2 < DIM; ++d2) Bk[d1][d2] = d1 == d2 ? fma(g[h][d1], mn[d2], dd) : g[h][d1] * mn[d2];
                        Bk[d1][Pc] = pN[d1];
                    }
                    double s = fma(cu, up[r], nuN);
                    if constexpr (FLOW) s = fma(ndl, dn[r], s) - vgk[h];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) Bk[Pc][d] = FLOW ? fma(s, rin[d], riVn * g[h][d]) : s * rin[d];
                    Bk[Pc][Pc] = gnk[h] * ppr;
                    // the 32 blocks go to L2 by consecutive entries: one reduction of the warp covers
                    // 128 bytes of each block instead of 8 bytes of 32 blocks (a quarter of the sectors)
#pragma unroll
                    for (int i = 0; i < T::BB; ++i) sblk[lane * T::STRIDE + i] = Bk[i / B][i % B];
                    __syncwarp();
                    auto reduce = [&](const int turn) {
#pragma unroll
                        for (int j = 0; j < T::BB; ++j) {
                            const int idx = j * 32 + lane, blk = idx / T::BB, ent = idx - blk * T::BB;
                            const double v = sblk[blk * T::STRIDE + ent];
                            const int32_t a0 = __shfl_sync(0xffffffffu, ql[r], blk), a1 = __shfl_sync(0xffffffffu, qh[r], blk);
                            if (SPLIT && ((blk >> 1) & 1) != turn) continue;
                            if (a0 >= 0) atomicAdd(vals + (int64_t)a0 * T::BB + ent, v);
                            if (a1 >= 0) atomicAdd(vals + (int64_t)a1 * T::BB + ent, flip_sign(v));
                        }
                        __syncwarp();
                    };
                    reduce(0);
                    if constexpr (SPLIT) reduce(1);
                }
            }
        }
        // the next axis updates rows of this one from other lanes: order the reductions
        __syncwarp();
    }
    if (!valid) return;
    if (!ok) atomicOr(A.err, 1);
    // ---- mass (implicit Euler) and source parts of this lane's corners
    if (tr || (def && P.hasSource)) {
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            const double vr = (AFFINE ? vol : sv[(l0 + k) * EPW]) * rho;
            const int c = k ? c1 : c0;
            if (def) {
                double* __restrict__ dk = A.D + (int64_t)(k ? nd1 : nd0) * B;
#pragma unroll
                for (int f = 0; f < DIM; ++f) {
                    double v = 0.0;
                    if (P.hasSource) v -= P.src[f] * vr;
                    if (tr) v = (su[(f * NSH + l0 + k) * EPW] * vr - so[(f * NSH + l0 + k) * EPW] * vr) + v * P.dt;
                    atomicAdd(dk + f, v);
                }
            }
            if (JAC && tr) {
                const int32_t q = __ldg(A.elemBlk + (int64_t)e * NSH * NSH + c * NSH + c);
                if (NSFV1_IN_RANGE(q, A.nnzb, A.err)) {
                    double* p = reinterpret_cast<double*>(A.vals) + (int64_t)q * (B * B);
#pragma unroll
                    for (int d = 0; d < DIM; ++d) atomicAdd(p + d * B + d, vr);
                }
            }
        }
    }
}

}  // namespace nsfv1

// nsfv1_simplex.cuh -- FP64 assembly of triangles and tetrahedra for the plain Navier-Stokes
// flag set (plain_params), one thread per element.
//
// The FP64 pipe bounds it (one warp instruction every 19 clocks per SM). On a simplex
// the gradients of every function and shape are constants of the element, so they, the
// symmetric gradient of the viscous flux and the pressure gradient are formed once instead
// of per SCVF; interpolation at an SCVF is a multiple of the corner sum plus a multiple
// of its edge's pair; normals and distances are combinations of the edge vectors; the LPS
// exit is the corner with the largest (v . grad N_k) / N_k, which is |v| / L_up (no square
// root, no cross-multiplied divisions); |v| / L of the full upwind takes one reciprocal square root
// per length; and 1 / dt is one division per element. The element's defect is summed
// in registers: dim + 1 reductions per corner instead of 2 (dim + 1) per SCVF and dim per
// corner. Jacobian blocks go through shared memory to the reductions as in nsfv1_tensor.cuh.
// Measured, general kernels (nsfv1_elem.cuh) before -> here: 2 x 1024^2 triangles, transient, full upwind +
// FIELDS, defect 2.73 -> 1.38 ms (676 -> 325 FP64 instructions a triangle); 6 x 24^3 tetrahedra, full +
// FLOW, defect 2.34 -> 1.25, Jacobian 2.94 -> 2.45, both 4.13 -> 2.80 ms.
// Registers: the launch bounds cost the tetrahedral Jacobian 200 bytes of spills with FLOW (48 with FIELDS)
// at 255 registers and the FLOW triangles 24 bytes.
#pragma once
#include "nsfv1_asm_common.cuh"
#include "nsfv1_tensor.cuh"

namespace nsfv1 {

template <int DIM>
struct Simp {
    static constexpr int ROID = DIM == 2 ? ROID_TRIANGLE : ROID_TETRAHEDRON;
    static constexpr int NSH = DIM + 1, B = DIM + 1, BB = B * B, STRIDE = BB | 1;
    // shape values at an SCVF's integration point: its edge's corners, the others
    static constexpr double NE = DIM == 2 ? 5.0 / 12.0 : 17.0 / 48.0, NO = DIM == 2 ? 1.0 / 6.0 : 7.0 / 48.0;
    static constexpr int smem_bytes(const bool jac, const int threads) { return jac ? threads * STRIDE * (int)sizeof(double) : 0; }
};

template <int DIM, bool JAC, bool FLOW>
__global__ void __launch_bounds__(kThreads, DIM == 2 ? (JAC ? 3 : 4) : 2) k_simplex(const DiscParams P, const AsmArgs A) {
    using T = Simp<DIM>;
    using R = Ref<T::ROID>;
    constexpr int NSH = T::NSH, B = T::B, Pc = DIM;
    extern __shared__ double smem[];
    const bool tr = P.transient != 0, def = !JAC || A.D != nullptr;
    const int lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool valid = t < A.count;
    if (!JAC && !valid) return;
    const int32_t e = __ldg(A.elems + (valid ? t : (int64_t)A.count - 1));
    if (A.elemInst && !__ldg(A.instActive + __ldg(A.elemInst + e))) valid = false;
    if (JAC ? !__any_sync(0xffffffffu, valid) : !valid) return;
    int32_t node[NSH];
#pragma unroll
    for (int k = 0; k < NSH; ++k) {
        node[k] = __ldg(A.conn + (int64_t)e * NSH + k);
        if (!NSFV1_IN_RANGE(node[k], A.nNodes, A.err)) { node[k] = 0; valid = false; }
    }
    double x[NSH][DIM], u[B][NSH], uo[DIM][NSH];
#pragma unroll
    for (int k = 0; k < NSH; ++k) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) x[k][d] = __ldg(A.coords + (int64_t)node[k] * DIM + d);
#pragma unroll
        for (int f = 0; f < B; ++f) u[f][k] = __ldg(A.U + (int64_t)node[k] * B + f);
    }
    if (tr && def)
#pragma unroll
        for (int k = 0; k < NSH; ++k)
#pragma unroll
            for (int d = 0; d < DIM; ++d) uo[d][k] = __ldg(A.Uold + (int64_t)node[k] * B + d);
    const double nu = A.nuElem ? __ldg(A.nuElem + e) : P.nu;
    const double rho = P.rho, mnr = -1.0 * nu * rho;
    double irho = 1.0, idt = 0.0;
    if (rho != 1.0) irho = 1.0 / rho;
    if (tr) idt = 1.0 / P.dt;
    const double js = tr ? P.dt : 1.0;
    const int upw = P.convUpwind;
    bool ok = true;

    // ---- element: gradients of the shapes, SCV volume
    double g[NSH][DIM], vol, edge[DIM == 2 ? 3 : 1][DIM];   // the triangle's edge vectors (edge 2: from 2 to 0)
    {
        double E[DIM][DIM], C[DIM][DIM], det = 0.0;
        if constexpr (DIM == 2) {
#pragma unroll
            for (int d = 0; d < 2; ++d) {
#pragma unroll
                for (int c = 0; c < 3; ++c) edge[c][d] = x[(c + 1) % 3][d] - x[c][d];
                E[0][d] = edge[0][d];
                E[1][d] = -edge[2][d];
            }
        } else {
#pragma unroll
            for (int c = 0; c < DIM; ++c)
#pragma unroll
                for (int d = 0; d < DIM; ++d) E[c][d] = x[c + 1][d] - x[0][d];
        }
        if constexpr (DIM == 3) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int p = (c + 1) % 3, q = (c + 2) % 3, d1 = (d + 1) % 3, d2 = (d + 2) % 3;
                    C[c][d] = E[p][d1] * E[q][d2] - E[p][d2] * E[q][d1];
                }
        } else {
            C[0][0] = E[1][1]; C[0][1] = -E[1][0];
            C[1][0] = -E[0][1]; C[1][1] = E[0][0];
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) det = fma(E[0][d], C[0][d], det);
        vol = fabs(det) * (DIM == 2 ? 1.0 / 6.0 : 1.0 / 24.0);
        const double id = 1.0 / det;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            double s = 0.0;
#pragma unroll
            for (int c = 0; c < DIM; ++c) { g[c + 1][d] = C[c][d] * id; s += g[c + 1][d]; }
            g[0][d] = -s;
        }
    }
    const double harea = 0.5 * vol * vol;
    // ---- corner sums and gradients of the functions
    double sum[B], base[DIM], S[DIM][DIM], gv[DIM][DIM], trace = 0.0;
    {
        double gp[DIM];
#pragma unroll
        for (int f = 0; f < B; ++f) {
            double s = u[f][0];
#pragma unroll
            for (int k = 1; k < NSH; ++k) s += u[f][k];
            sum[f] = s * T::NO;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                double a = 0.0;
#pragma unroll
                for (int k = 1; k < NSH; ++k) a = fma(u[f][k] - u[f][0], g[k][d], a);
                if (f < DIM) gv[f < DIM ? f : 0][d] = a;
                else gp[d] = a;
            }
        }
        // the constant part of the stabilised velocity's right-hand side, and the viscous stress
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            base[d] = fma(-irho, gp[d], P.hasSource ? P.src[d] : 0.0);
            trace += gv[d][d];
#pragma unroll
            for (int q = 0; q < DIM; ++q) S[d][q] = mnr * (gv[d][q] + gv[q][d]);
        }
        if (tr && def)
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                double s = uo[d][0];
#pragma unroll
                for (int k = 1; k < NSH; ++k) s += uo[d][k];
                base[d] = fma(T::NO * idt, s, base[d]);
            }
    }
    const double ndt = (T::NE - T::NO) * idt;
    double acc[B][NSH];   // the element's defect
#pragma unroll
    for (int f = 0; f < B; ++f)
#pragma unroll
        for (int k = 0; k < NSH; ++k) acc[f][k] = 0.0;

#pragma unroll
    for (int ip = 0; ip < R::nip; ++ip) {
        const int i = R::edge(ip, 0), j = R::edge(ip, 1);
        // z = edge midpoint -> centre; n from i to j
        double z[DIM], n[DIM], eij[DIM];
        if constexpr (DIM == 2) {
            const int k = 3 - i - j;   // edge j runs from j to k, edge k from k to i
#pragma unroll
            for (int d = 0; d < 2; ++d) {
                eij[d] = edge[ip][d];
                z[d] = (edge[j][d] - edge[k][d]) * (1.0 / 6.0);
            }
            n[0] = z[1];
            n[1] = -z[0];
        } else {
            // the faces at the edge: i, j and one of the two other corners
            const int f1 = R::edge_face(ip, 0);
            int k = -1, l = -1;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c != i && c != j) {
                    bool in1 = false;
#pragma unroll
                    for (int q = 0; q < 3; ++q) in1 = in1 || R::side(f1, q) == c;
                    if (in1) k = c;
                    else l = c;
                }
            double w[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                z[d] = (x[k][d] - x[i][d]) + (x[l][d] - x[j][d]);   // 4 z
                w[d] = x[l][d] - x[k][d];                           // 3 (second face centre - first)
                eij[d] = x[j][d] - x[i][d];
            }
            n[0] = (z[1] * w[2] - z[2] * w[1]) * (1.0 / 24.0);
            n[1] = (z[2] * w[0] - z[0] * w[2]) * (1.0 / 24.0);
            n[2] = (z[0] * w[1] - z[1] * w[0]) * (1.0 / 24.0);
#pragma unroll
            for (int d = 0; d < 3; ++d) z[d] *= 0.25;
        }
        double val[B], nn = 0.0, vv = 0.0, Vn = 0.0, ds = 0.0;
#pragma unroll
        for (int f = 0; f < B; ++f) val[f] = fma(T::NE - T::NO, u[f][i] + u[f][j], sum[f]);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            nn = fma(n[d], n[d], nn);
            vv = fma(val[d], val[d], vv);
            Vn = fma(n[d], val[d], Vn);
            if (DIM == 3) ds = fma(z[d], z[d], ds);
        }
        if (DIM == 2) ds = nn;
        const double nuL = (nu * nn) * (1.0 / fma(0.375 * ds, nn, harea));
        // rate of the barycentric coordinates along v: r_k = v . grad N_k (LPS; FLOW's Jacobian)
        double r[NSH];
#pragma unroll
        for (int k = 0; k < NSH; ++k) r[k] = 0.0;
        if (upw == UPW_LPS || (FLOW && JAC)) {
            double s = 0.0;
#pragma unroll
            for (int k = 1; k < NSH; ++k) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) r[k] = fma(g[k][d], val[d], r[k]);
                s += r[k];
            }
            r[0] = -s;
        }
        // ---- upwind (and downwind): velocity, shapes, ncl = |v| / L_up, ndl = |v| / (L_down + L_up)
        double upv[DIM], dnv[DIM], up[NSH], dn[NSH], ncl, ndl = 0.0;
        const double norm = (upw == UPW_NO || (FLOW && upw == UPW_FULL) || vv < 1.01e-28) ? speed(vv) : 1.0;
        if (upw == UPW_FULL) {
            // (sign tests on the bits: a comparison is an FP64 instruction)
            const bool fr = __double_as_longlong(Vn) > 0;                          // upwind corner i, else j
            const bool df = __double_as_longlong(flip_sign(Vn)) > 0;               // downwind corner i, else j (a zero flux: j for both)
            // twice the vector from the corner to the integration point: edge midpoint -> integration
            // point is z / 2 (2D), 7/12 z (3D)
            double l2 = 0.0, d2 = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double c = DIM == 2 ? z[d] : (7.0 / 6.0) * z[d], me = flip_sign(eij[d]);
                const double a = c + (fr ? eij[d] : me);
                l2 = fma(a, a, l2);
                if constexpr (FLOW) {
                    const double w = c + (df ? eij[d] : me);
                    d2 = fma(w, w, d2);
                }
                upv[d] = fr ? u[d][i] : u[d][j];
                dnv[d] = df ? u[d][i] : u[d][j];
            }
#pragma unroll
            for (int k = 0; k < NSH; ++k) {
                up[k] = k == i ? (fr ? 1.0 : 0.0) : k == j ? (fr ? 0.0 : 1.0) : 0.0;
                dn[k] = k == i ? (df ? 1.0 : 0.0) : k == j ? (df ? 0.0 : 1.0) : 0.0;
            }
            if constexpr (FLOW) {
                const double ru = rsqrt(l2);
                ncl = 2.0 * (norm * ru);
                ndl = 2.0 * norm / fma(d2, rsqrt(d2), l2 * ru);
            } else {
                // |v| / L = 2 v^2 / sqrt(v^2 l2); the product outside the normal range: one factor at a time
                const double p = vv * l2;
                if (p > 1e-280 && p < 1e280) ncl = 2.0 * vv * rsqrt(p);
                else ncl = 2.0 * speed(vv) * rsqrt(l2);
            }
        } else if (upw == UPW_LPS && !(norm < 1e-14)) {
            // the ray along -v leaves where the first coordinate N_k - s r_k vanishes
            double bu = 0.0, bd = 0.0;
            int ku = -1, kd = -1;
#pragma unroll
            for (int k = 0; k < NSH; ++k) {
                const double q = r[k] * (k == i || k == j ? 1.0 / T::NE : 1.0 / T::NO);
                if (q > bu) { bu = q; ku = k; }
                if (FLOW && -q > bd) { bd = -q; kd = k; }
            }
            if (ku < 0) ok = false;   // a velocity that is not a number
            ncl = bu;
            const double s = 1.0 / bu, sd = FLOW ? 1.0 / bd : 0.0;
            if constexpr (FLOW) ndl = 1.0 / (s + sd);
#pragma unroll
            for (int k = 0; k < NSH; ++k) {
                const double N = k == i || k == j ? T::NE : T::NO;
                up[k] = k == ku ? 0.0 : fma(-s, r[k], N);
                dn[k] = FLOW ? (k == kd ? 0.0 : fma(sd, r[k], N)) : 0.0;
            }
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                upv[d] = 0.0; dnv[d] = 0.0;
#pragma unroll
                for (int k = 0; k < NSH; ++k) {
                    upv[d] = fma(up[k], u[d][k], upv[d]);
                    if constexpr (FLOW) dnv[d] = fma(dn[k], u[d][k], dnv[d]);
                }
            }
        } else {
            const bool zero = upw == UPW_LPS;
#pragma unroll
            for (int d = 0; d < DIM; ++d) upv[d] = dnv[d] = zero ? 0.0 : val[d];
#pragma unroll
            for (int k = 0; k < NSH; ++k) up[k] = dn[k] = zero ? 0.0 : (k == i || k == j ? T::NE : T::NO);
            ncl = norm;
            if constexpr (FLOW) ndl = 0.5 * norm;
        }
        double diag = nuL + ncl;
        if (tr) diag += idt;
        const double idiag = 1.0 / diag, cu = FLOW ? ncl - ndl : ncl;
        if (def) {
            double cont = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                double rhs = base[d];
                if (tr) rhs = fma(ndt, uo[d][i] + uo[d][j], rhs);
                rhs = fma(nuL, val[d], rhs);
                rhs = fma(cu, upv[d], rhs);
                double fl = fma(upv[d], rho * Vn, val[Pc] * n[d]);
                if constexpr (FLOW) {
                    double cv = 0.0;
#pragma unroll
                    for (int q = 0; q < DIM; ++q) cv = fma(val[q], gv[d][q], cv);
                    rhs = fma(ndl, dnv[d], rhs) + (val[d] * trace - cv);
                }
                cont = fma(rhs, n[d], cont);
#pragma unroll
                for (int q = 0; q < DIM; ++q) fl = fma(S[d][q], n[q], fl);
                acc[d][i] += fl;
                acc[d][j] -= fl;
            }
            cont *= rho * idiag;
            acc[Pc][i] += cont;
            acc[Pc][j] -= cont;
        }
        if constexpr (JAC) {
            const double m = mnr * js, ri = rho * idiag * js, pw = Vn * rho * js, riVn = ri * Vn, ppr = -(idiag * js);
            double mn[DIM], rin[DIM], pn[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) { mn[d] = m * n[d]; rin[d] = ri * n[d]; pn[d] = js * n[d]; }
            double* sblk = smem + (threadIdx.x >> 5) * (32 * T::STRIDE);
            double* __restrict__ vals = reinterpret_cast<double*>(A.vals);
#pragma unroll
            for (int k = 0; k < NSH; ++k) {
                const double N = k == i || k == j ? T::NE : T::NO;
                int32_t q0 = __ldg(A.elemBlk + (int64_t)e * NSH * NSH + i * NSH + k), q1 = __ldg(A.elemBlk + (int64_t)e * NSH * NSH + j * NSH + k);
                if (!valid || !NSFV1_IN_RANGE(q0, A.nnzb, A.err)) q0 = -1;
                if (!valid || !NSFV1_IN_RANGE(q1, A.nnzb, A.err)) q1 = -1;
                double Bk[B][B], gn = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) gn = fma(g[k][d], n[d], gn);
                const double dd = fma(up[k], pw, m * gn);
#pragma unroll
                for (int d1 = 0; d1 < DIM; ++d1) {
#pragma unroll
                    for (int d2 = 0; d2 < DIM; ++d2) Bk[d1][d2] = d1 == d2 ? fma(g[k][d1], mn[d2], dd) : g[k][d1] * mn[d2];
                    Bk[d1][Pc] = N * pn[d1];
                }
                double s = fma(cu, up[k], nuL * N);
                if constexpr (FLOW) s = fma(ndl, dn[k], s) - r[k];
#pragma unroll
                for (int d = 0; d < DIM; ++d) Bk[Pc][d] = FLOW ? fma(s, rin[d], riVn * g[k][d]) : s * rin[d];
                Bk[Pc][Pc] = gn * ppr;
#pragma unroll
                for (int c = 0; c < T::BB; ++c) sblk[lane * T::STRIDE + c] = Bk[c / B][c % B];
                __syncwarp();
#pragma unroll
                for (int c = 0; c < T::BB; ++c) {
                    const int idx = c * 32 + lane, blk = idx / T::BB, ent = idx - blk * T::BB;
                    const double v = sblk[blk * T::STRIDE + ent];
                    const int32_t a0 = __shfl_sync(0xffffffffu, q0, blk), a1 = __shfl_sync(0xffffffffu, q1, blk);
                    if (a0 >= 0) atomicAdd(vals + (int64_t)a0 * T::BB + ent, v);
                    if (a1 >= 0) atomicAdd(vals + (int64_t)a1 * T::BB + ent, flip_sign(v));
                }
                __syncwarp();
            }
        }
    }
    if (!valid) return;
    if (!ok) atomicOr(A.err, 1);
    // ---- the element's defect with its mass (implicit Euler) and source parts; the mass blocks
    const double vr = vol * rho;
#pragma unroll
    for (int k = 0; k < NSH; ++k) {
        if (def) {
            double* __restrict__ dk = A.D + (int64_t)node[k] * B;
#pragma unroll
            for (int f = 0; f < B; ++f) {
                double v = acc[f][k];
                if (f < DIM && P.hasSource) v = fma(-P.src[f < DIM ? f : 0], vr, v);
                if (tr) {
                    v *= js;
                    if (f < DIM) v = fma(u[f][k] - uo[f < DIM ? f : 0][k], vr, v);
                }
                atomicAdd(dk + f, v);
            }
        }
        if (JAC && tr) {
            const int32_t q = __ldg(A.elemBlk + (int64_t)e * NSH * NSH + k * NSH + k);
            if (NSFV1_IN_RANGE(q, A.nnzb, A.err)) {
                double* p = reinterpret_cast<double*>(A.vals) + (int64_t)q * T::BB;
#pragma unroll
                for (int d = 0; d < DIM; ++d) atomicAdd(p + d * B + d, vr);
            }
        }
    }
}

}  // namespace nsfv1

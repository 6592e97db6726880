// Barrier energy, body-space gradient and 12x12 pair Hessian per constraint,
// with the rigid-pose chain rule folded in, and their deterministic assembly
// into a per-body gradient and a 6x6 block-sparse Hessian.
//
// Replaces DistanceBarrierRBProblem::compute_barrier_term
// (src/problems/distance_barrier_rb_problem.cpp:1299-1399): the ipc-toolkit
// constraint potentials (log barrier of the squared distance shifted by
// dmin^2, src/opt/distance_barrier_constraint.tpp:11-17; EE mollifier),
// apply_chain_rule (:1182-1248, including project_to_psd of the 12x12),
// local_hessian_to_global_triplets (:1157-1179) and merge_derivative_storage
// (:1260-1297).
//
// Derivation used by k_barrier_local.  With X the constraint's vertex
// positions and x the two bodies' 6-dof poses, X_i = R_b v_i + p_b and
// J_i = dX_i/dx_b = [I | D_i], D_i[:, k] = (dR/dtheta_k) v_i.
//  * PT / EE: d = u^2 / D with u = (A x B).w and D = |A x B|^2, where
//    A, B, w are signed sums of the vertices (coefficients alpha, beta,
//    gamma).  grad u = {alpha_i (B x w) + beta_i (w x A) + gamma_i n},
//    grad D = {2 alpha_i (B x n) + 2 beta_i (n x A)}; the Hessians are
//    Gram(dn) terms and skew bilinear blocks [s_ij]x between vertices i != j.
//  * PE: d = |a x b|^2 / |e|^2, the same pieces with a Gram(de) term.
//  * PP: d = |w|^2.
// f = weight * m(D) * b(d - dmin^2) (m = 1 except mollified EE), so the body
// Hessian is  sum of outer products of the body-space gradients of the basic
// scalars + Gram terms + skew pair blocks + the curvature term
// sum_i grad_Xi f . d2X_i/dtheta2.  It is then projected to the PSD cone,
// V max(L, 0) V^T (local_terms.cuh).
#include <algorithm>

#include "common.cuh"
#include "geometry_rn.cuh"
#include "local_terms.cuh"
#include "rotation.cuh"
#include "sort.cuh"

namespace rigc {

// ---------------------------------------------------------------------------
// per-body frames (R, dR, d2R) and positions

__global__ void k_body_frames(const double* __restrict__ x, int nb, double* __restrict__ frames)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    double t[3] = { x[6 * b + 3], x[6 * b + 4], x[6 * b + 5] };
    double F[kFrameDoubles];
    body_frame(t, F);
    double* out = frames + (size_t)b * 96;
#pragma unroll
    for (int i = 0; i < kFrameDoubles; i++) out[i] = F[i];
    out[90] = x[6 * b];
    out[91] = x[6 * b + 1];
    out[92] = x[6 * b + 2];
}

// ---------------------------------------------------------------------------

struct BarrierArgs {
    const double* rest;
    const double* frames;
    const int* ctype;
    const int* cverts;
    const int* cbodies;
    const double* cweight;
    const double* ceps;
    int64_t n;
    double dhat, dmin;
    int flags;
    double* energy;   // n
    double* grad;     // n x 12
    double* blocks;   // n x 4 x 36 (blocks (0,0) (0,1) (1,0) (1,1))
    double* hess;     // optional n x 144 (full local Hessian)
    // index limits checked on the device when check_nv >= 0 (callers whose
    // constraint arrays were not validated on the host): a constraint with a
    // type, vertex or body index out of range reads nothing and gets NaN
    // outputs
    int check_nb = 0;
    int64_t check_nv = -1;
};

// the index check of a constraint (see BarrierArgs::check_nv)
static __device__ bool constraint_in_range(const BarrierArgs& a, int64_t ci)
{
    const int type = a.ctype[ci];
    if (type < 0 || type > 3) return false;
    const int nvc = type == 0 ? 2 : (type == 1 ? 3 : 4);
    for (int i = 0; i < 2; i++) {
        const int b = a.cbodies[2 * ci + i];
        if (b < 0 || b >= a.check_nb) return false;
    }
    for (int i = 0; i < nvc; i++) {
        const int v = a.cverts[4 * ci + i];
        if (v < 0 || (int64_t)v >= a.check_nv) return false;
    }
    return true;
}

__device__ __forceinline__ int local_body_of(int type, int i)
{
    if (type == 2) return i < 2 ? 0 : 1;
    return i == 0 ? 0 : 1;
}

// A mollified EE constraint whose closest features are endpoints (kept as EE
// by the constraint set because the edges are nearly parallel): f = w m(D)
// b(d - dmin^2) with D = |A x B|^2 of the two edges and d the point-point or
// point-edge squared distance of the closest features.  Vertex-space
// gradients and 3x3 Hessian blocks in closed form:
//   grad D_i = 2 M_i^T n, M_i = alpha_i (-[B]x) + beta_i [A]x,
//   hess D_ij = 2 M_i^T M_j + 2 (beta_i alpha_j - alpha_i beta_j) [n]x,
// and the same for N = |a x b|^2 of a point-edge distance d = N / |e|^2, so the
// body Hessian is outer products of the body-space gradients, Gram terms, skew
// pair blocks and the curvature term, as barrier_build's: bound by FP64 issue,
// and most constraints of box-like bodies in contact end here (104 k of 163 k
// between 32 slabs).  J_i^T (.) J_j of the ten 3x3 vertex blocks took 2.20 ms
// there, with the other kinds, unprojected; this 1.34 ms (338 constraints
// between 27 cubes, one per lane: 256 -> 212 us).
static __device__ __noinline__ bool ee_endpoint_build(const BarrierArgs& a, int64_t ci, SMat H,
                                                      const Vtx* V, const double (*vrest)[3],
                                                      const int* lbody, const double* const* fr,
                                                      int dtype)
{
    const double weight = a.cweight[ci];
    int kind = 1, p = 0, q = 0, e0 = 0, e1 = 0;
    switch (dtype) {
    case EE_EA0_EB0: kind = 0; p = 0; q = 2; break;
    case EE_EA0_EB1: kind = 0; p = 0; q = 3; break;
    case EE_EA1_EB0: kind = 0; p = 1; q = 2; break;
    case EE_EA1_EB1: kind = 0; p = 1; q = 3; break;
    case EE_EA_EB0: p = 2; e0 = 0; e1 = 1; break;
    case EE_EA_EB1: p = 3; e0 = 0; e1 = 1; break;
    case EE_EA0_EB: p = 0; e0 = 2; e1 = 3; break;
    default: p = 1; e0 = 2; e1 = 3; break;
    }
    const double alD[4] = { -1, 1, 0, 0 }, beD[4] = { 0, 0, -1, 1 };
    double A[3], B[3], n[3];
    for (int j = 0; j < 3; j++) {
        A[j] = V[1].X[j] - V[0].X[j];
        B[j] = V[3].X[j] - V[2].X[j];
    }
    cross(A, B, n);
    const double Dm = dot(n, n);
    double gD[4][3], gd[4][3];
    {
        double Bn[3], nA[3];
        cross(B, n, Bn);
        cross(n, A, nA);
        for (int i = 0; i < 4; i++)
            for (int j = 0; j < 3; j++) {
                gD[i][j] = 2 * (alD[i] * Bn[j] + beD[i] * nA[j]);
                gd[i][j] = 0;
            }
    }
    double d, N = 0, De = 1;
    double pa[3], pb[3], c[3], e[3];
    double alE[4] = { 0, 0, 0, 0 }, beE[4] = { 0, 0, 0, 0 }, gaE[4] = { 0, 0, 0, 0 };
    double gN[4][3], gE[4][3];
    if (kind == 0) {
        double w[3];
        for (int j = 0; j < 3; j++) w[j] = V[p].X[j] - V[q].X[j];
        d = dot(w, w);
        for (int j = 0; j < 3; j++) {
            gd[p][j] = 2 * w[j];
            gd[q][j] = -2 * w[j];
        }
    } else {
        alE[p] = -1; alE[e0] = 1; beE[p] = -1; beE[e1] = 1; gaE[e0] = -1; gaE[e1] = 1;
        for (int j = 0; j < 3; j++) {
            pa[j] = V[e0].X[j] - V[p].X[j];
            pb[j] = V[e1].X[j] - V[p].X[j];
            e[j] = V[e1].X[j] - V[e0].X[j];
        }
        cross(pa, pb, c);
        N = dot(c, c);
        De = dot(e, e);
        d = N / De;
        double bc[3], ca[3];
        cross(pb, c, bc);
        cross(c, pa, ca);
        for (int i = 0; i < 4; i++)
            for (int j = 0; j < 3; j++) {
                gN[i][j] = 2 * (alE[i] * bc[j] + beE[i] * ca[j]);
                gE[i][j] = 2 * gaE[i] * e[j];
                gd[i][j] = gN[i][j] / De - N / (De * De) * gE[i][j];
            }
    }
    // barrier of the shifted squared distance and the mollifier
    const double s = 2 * a.dmin * a.dhat + a.dhat * a.dhat;
    const double dd = d - a.dmin * a.dmin;
    double bv = 0, b1 = 0, b2 = 0;
    bool active = dd < s;
    if (dd <= 0.0) {
        bv = INFINITY;
        active = false;
    } else if (active) {
        double lg = log(dd / s);
        double dm = dd - s;
        bv = -dm * dm * lg;
        b1 = (s - dd) * (2 * lg - s / dd + 1);
        double sd = s / dd;
        b2 = (sd + 2) * sd - 2 * lg - 3;
    }
    double m = 1, m1 = 0, m2 = 0;
    if (Dm < a.ceps[ci]) {
        double ie = 1.0 / a.ceps[ci];
        double xe = Dm * ie;
        m = (2 - xe) * xe;
        m1 = (2 - 2 * xe) * ie;
        m2 = -2 * ie * ie;
    }
    if (a.energy) a.energy[ci] = weight * m * bv;
    const bool want_g = (a.flags & (RIGC_GRAD | RIGC_HESS)) != 0;
    const bool want_h = (a.flags & RIGC_HESS) != 0;
    if (!active) {
        if (a.grad)
            for (int k = 0; k < 12; k++) a.grad[ci * 12 + k] = 0;
        if (a.blocks && want_h)
            for (int k = 0; k < 144; k++) a.blocks[ci * 144 + k] = 0;
        if (a.hess && want_h)
            for (int k = 0; k < 144; k++) a.hess[ci * 144 + k] = 0;
        return false;
    }
    if (!want_g) return false;
    double gv[4][3];
    for (int i = 0; i < 4; i++)
        for (int j = 0; j < 3; j++) gv[i][j] = weight * (m * b1 * gd[i][j] + bv * m1 * gD[i][j]);
    double G[12];
    to_body(V, lbody, 4, gv, G);
    if (a.grad)
        for (int k = 0; k < 12; k++) a.grad[ci * 12 + k] = G[k];
    if (!want_h) return false;

    H.clear();
    const double cd = weight * m * b1, cD = weight * bv * m1;  // on hess d, hess D
    const double kdd = weight * m * b2, kdD = weight * m1 * b1, kDD = weight * bv * m2;
    double M[4][9];
    // M_i = alpha_i (-[B]x) + beta_i [A]x (dn/dX_i, likewise of c = pa x pb)
    auto skew_of = [](double sa, const double* Bv, double sb, const double* Av, double* Mi) {
        const double v0 = -sa * Bv[0] + sb * Av[0], v1 = -sa * Bv[1] + sb * Av[1], v2 = -sa * Bv[2] + sb * Av[2];
        Mi[0] = 0; Mi[1] = -v2; Mi[2] = v1;
        Mi[3] = v2; Mi[4] = 0; Mi[5] = -v0;
        Mi[6] = -v1; Mi[7] = v0; Mi[8] = 0;
    };
    for (int i = 0; i < 4; i++) skew_of(alD[i], B, beD[i], A, M[i]);
    add_gram(H, 2 * cD, V, lbody, 4, M);
    double gr[3][kRed];
    to_body(V, lbody, 4, gD, G);
    reduce12(G, gr[2]);
    if (kind == 0) {
        // d = |w|^2: hess = 2 (dw)^T (dw)
        to_body(V, lbody, 4, gd, G);
        reduce12(G, gr[1]);
        add_quadratic(H, kdd, kdD, kDD, gr[1], gr[2]);
        for (int i = 0; i < 4; i++) {
            for (int k = 0; k < 9; k++) M[i][k] = 0;
            M[i][0] = M[i][4] = M[i][8] = i == p ? 1.0 : (i == q ? -1.0 : 0.0);
        }
        add_gram(H, 2 * cd, V, lbody, 4, M);
    } else {
        // grad d = gN / De - N / De^2 gE,
        // hess d = (1/De) H_N - (1/De^2)(gN gE + gE gN) + (2N/De^3) gE gE - (N/De^2) H_E
        const double pn = 1 / De, pe = -N / (De * De);
        to_body(V, lbody, 4, gN, G);
        reduce12(G, gr[0]);
        to_body(V, lbody, 4, gE, G);
        reduce12(G, gr[1]);
        double gdr[kRed];  // reduced body gradient of d
        for (int k = 0; k < kRed; k++) gdr[k] = pn * gr[0][k] + pe * gr[1][k];
        add_quadratic(H, kdd, kdD, kDD, gdr, gr[2]);
        add_quadratic(H, 0, -cd / (De * De), 2 * cd * N / (De * De * De), gr[0], gr[1]);
        for (int i = 0; i < 4; i++) skew_of(alE[i], pb, beE[i], pa, M[i]);
        add_gram(H, 2 * cd / De, V, lbody, 4, M);
        for (int i = 0; i < 4; i++) {
            for (int k = 0; k < 9; k++) M[i][k] = 0;
            M[i][0] = M[i][4] = M[i][8] = gaE[i];
        }
        add_gram(H, 2 * cd * pe, V, lbody, 4, M);
    }
    for (int i = 0; i < 4; i++)
        for (int j = i + 1; j < 4; j++) {
            const double kD = 2 * cD * (beD[i] * alD[j] - alD[i] * beD[j]);
            const double kN = kind == 1 ? 2 * cd / De * (beE[i] * alE[j] - alE[i] * beE[j]) : 0.0;
            if (kD == 0 && kN == 0) continue;
            double sv[3];
            for (int k = 0; k < 3; k++) sv[k] = kD * n[k] + (kind == 1 ? kN * c[k] : 0.0);
            add_skew_pair(H, V[i], lbody[i], V[j], lbody[j], sv);
        }
    add_curvature(H, fr, lbody, 4, vrest, gv);
    return true;
}

// Energy, gradient and (reduced) unprojected body Hessian of constraint ci
// into H; returns true when H holds a Hessian to project and
// write, false when every output of the constraint is already written.
static __device__ __noinline__ bool barrier_build(const BarrierArgs& a, int64_t ci, SMat H)
{
    if (a.check_nv >= 0 && !constraint_in_range(a, ci)) {
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        if (a.energy) a.energy[ci] = nan;
        if (a.grad)
            for (int k = 0; k < 12; k++) a.grad[ci * 12 + k] = nan;
        if (a.flags & RIGC_HESS) {
            if (a.blocks)
                for (int k = 0; k < 144; k++) a.blocks[ci * 144 + k] = nan;
            if (a.hess)
                for (int k = 0; k < 144; k++) a.hess[ci * 144 + k] = nan;
        }
        return false;
    }
    const int type = a.ctype[ci];
    const int nvc = type == 0 ? 2 : (type == 1 ? 3 : 4);
    const double weight = a.cweight[ci];
    int lbody[4];
    const double* fr[2];
    int bod[2] = { a.cbodies[2 * ci], a.cbodies[2 * ci + 1] };
    fr[0] = a.frames + (size_t)bod[0] * 96;
    fr[1] = a.frames + (size_t)bod[1] * 96;
    Vtx V[4];
    double vrest[4][3];
    for (int i = 0; i < nvc; i++) {
        lbody[i] = local_body_of(type, i);
        int vi = a.cverts[4 * ci + i];
        const double* f = fr[lbody[i]];
        for (int j = 0; j < 3; j++) vrest[i][j] = a.rest[3 * (size_t)vi + j];
        const double* v = vrest[i];
        for (int j = 0; j < 3; j++) {
            V[i].X[j] = f[3 * j] * v[0] + f[3 * j + 1] * v[1] + f[3 * j + 2] * v[2] + f[90 + j];
            for (int k = 0; k < 3; k++) {
                const double* dR = f + 9 + 9 * k;
                V[i].D[j][k] = dR[3 * j] * v[0] + dR[3 * j + 1] * v[1] + dR[3 * j + 2] * v[2];
            }
        }
    }

    if (type == 2) {
        const int dt = ee_type_rn(V[0].X, V[1].X, V[2].X, V[3].X);
        if (dt != EE_EA_EB) return ee_endpoint_build(a, ci, H, V, vrest, lbody, fr, dt);
    }

    // coefficient patterns: A = sum alpha_i X_i, B = sum beta_i X_i, w = sum gamma_i X_i
    double al[4] = { 0, 0, 0, 0 }, be[4] = { 0, 0, 0, 0 }, ga[4] = { 0, 0, 0, 0 };
    double A[3], B[3], W[3], n[3];
    double d, u = 0, Dn = 0;
    if (type == 2) {        // EE: A = X1 - X0, B = X3 - X2, w = X2 - X0
        al[0] = -1; al[1] = 1; be[2] = -1; be[3] = 1; ga[0] = -1; ga[2] = 1;
    } else if (type == 3) { // FV: A = X2 - X1, B = X3 - X1, w = X0 - X1
        al[1] = -1; al[2] = 1; be[1] = -1; be[3] = 1; ga[0] = 1; ga[1] = -1;
    } else if (type == 1) { // EV: a = X1 - X0, b = X2 - X0 ; e = X2 - X1 (gamma)
        al[0] = -1; al[1] = 1; be[0] = -1; be[2] = 1; ga[1] = -1; ga[2] = 1;
    } else {                // VV: w = X0 - X1
        ga[0] = 1; ga[1] = -1;
    }
    for (int j = 0; j < 3; j++) {
        A[j] = 0; B[j] = 0; W[j] = 0;
        for (int i = 0; i < nvc; i++) {
            A[j] += al[i] * V[i].X[j];
            B[j] += be[i] * V[i].X[j];
            W[j] += ga[i] * V[i].X[j];
        }
    }
    double De = 0;
    if (type >= 2) {
        cross(A, B, n);
        u = dot(n, W);
        Dn = dot(n, n);
        d = u * u / Dn;
    } else if (type == 1) {
        cross(A, B, n);  // c = a x b
        Dn = dot(n, n);  // N = |c|^2
        De = dot(W, W);  // |e|^2
        d = Dn / De;
    } else {
        d = dot(W, W);
        n[0] = n[1] = n[2] = 0;
    }

    // barrier of the shifted squared distance
    const double s = 2 * a.dmin * a.dhat + a.dhat * a.dhat;
    const double dd = d - a.dmin * a.dmin;
    double bv = 0, b1 = 0, b2 = 0;
    bool active = dd < s;
    if (dd <= 0.0) {
        bv = INFINITY;
        active = false;
    } else if (active) {
        double lg = log(dd / s);
        double dm = dd - s;
        bv = -dm * dm * lg;
        b1 = (s - dd) * (2 * lg - s / dd + 1);
        double sd = s / dd;
        b2 = (sd + 2) * sd - 2 * lg - 3;
    }
    // EE mollifier m(D), D = |A x B|^2
    double m = 1, m1 = 0, m2 = 0;
    if (type == 2 && Dn < a.ceps[ci]) {
        double ie = 1.0 / a.ceps[ci];
        double xe = Dn * ie;
        m = (2 - xe) * xe;
        m1 = (2 - 2 * xe) * ie;
        m2 = -2 * ie * ie;
    }
    if (a.energy) a.energy[ci] = weight * m * bv;
    const bool want_g = (a.flags & (RIGC_GRAD | RIGC_HESS)) != 0;
    const bool want_h = (a.flags & RIGC_HESS) != 0;
    if (!active) {
        if (a.grad)
            for (int k = 0; k < 12; k++) a.grad[ci * 12 + k] = 0;
        if (a.blocks && want_h)
            for (int k = 0; k < 144; k++) a.blocks[ci * 144 + k] = 0;
        if (a.hess && want_h)
            for (int k = 0; k < 144; k++) a.hess[ci * 144 + k] = 0;
        return false;
    }
    if (!want_g) return false;

    // ---- basic scalars and their vertex-space gradients
    // g1: gradient of the first scalar (u, N or d), g2: of the second (D, |e|^2)
    double g1v[4][3], g2v[4][3];
    double c1, c2;  // grad d = c1 g1 + c2 g2
    if (type >= 2) {
        double Bw[3], wA[3], Bn[3], nA[3];
        cross(B, W, Bw);
        cross(W, A, wA);
        cross(B, n, Bn);
        cross(n, A, nA);
        for (int i = 0; i < 4; i++)
            for (int j = 0; j < 3; j++) {
                g1v[i][j] = al[i] * Bw[j] + be[i] * wA[j] + ga[i] * n[j];
                g2v[i][j] = 2 * (al[i] * Bn[j] + be[i] * nA[j]);
            }
        c1 = 2 * u / Dn;
        c2 = -u * u / (Dn * Dn);
    } else if (type == 1) {
        double bc[3], ca[3];
        cross(B, n, bc);
        cross(n, A, ca);
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) {
                g1v[i][j] = 2 * (al[i] * bc[j] + be[i] * ca[j]);
                g2v[i][j] = 2 * ga[i] * W[j];
            }
        c1 = 1 / De;
        c2 = -Dn / (De * De);
    } else {
        for (int j = 0; j < 3; j++) {
            g1v[0][j] = 2 * W[j];
            g1v[1][j] = -2 * W[j];
            g2v[0][j] = g2v[1][j] = 0;
        }
        c1 = 1;
        c2 = 0;
    }
    // f = weight * m * b(d):  grad f = P_g1 g1 + P_g2 g2
    const double wm = weight * m;
    // (the mollifier's gradient lies along grad D = g2, EE only)
    const double Pg1 = wm * b1 * c1;
    const double Pg2 = wm * b1 * c2 + (type == 2 ? weight * bv * m1 : 0.0);
    double gv[4][3];
    for (int i = 0; i < nvc; i++)
        for (int j = 0; j < 3; j++) gv[i][j] = Pg1 * g1v[i][j] + Pg2 * g2v[i][j];
    double G[12];
    to_body(V, lbody, nvc, gv, G);
    if (a.grad)
        for (int k = 0; k < 12; k++) a.grad[ci * 12 + k] = G[k];
    if (!want_h) return false;

    // ---- Hessian
    H.clear();
    double G12[2][kRed];
    to_body(V, lbody, nvc, g1v, G);
    reduce12(G, G12[0]);
    to_body(V, lbody, nvc, g2v, G);
    reduce12(G, G12[1]);
    // second-derivative coefficients of d in terms of (g1, g2) and the
    // Hessians of the basic scalars:
    //  PT/EE: hess d = (2/D) g1g1 + c1 H_u - (2u/D^2)(g1g2 + g2g1) + (2u^2/D^3) g2g2 + c2 H_D
    //  PE:    hess d = (1/De) H_N - (1/De^2)(g1g2 + g2g1) + (2N/De^3) g2g2 + c2 H_e
    //  PP:    hess d = H_w (Gram of dw)
    double duu, duD, dDD;
    if (type >= 2) {
        duu = 2 / Dn;
        duD = -2 * u / (Dn * Dn);
        dDD = 2 * u * u / (Dn * Dn * Dn);
    } else if (type == 1) {
        duu = 0;
        duD = -1 / (De * De);
        dDD = 2 * Dn / (De * De * De);
    } else {
        duu = duD = dDD = 0;
    }
    // f Hessian = P1 gd gd^T + P2 hess d + [EE] P3 g2g2 + P4 H_D + P5 (g2 gd^T + gd g2^T)
    const double P1 = wm * b2, P2 = wm * b1;
    const double P3 = type == 2 ? weight * bv * m2 : 0.0;
    const double P4 = type == 2 ? weight * bv * m1 : 0.0;
    const double P5 = type == 2 ? weight * m1 * b1 : 0.0;
    const double a11 = P1 * c1 * c1 + P2 * duu;
    const double a12 = P1 * c1 * c2 + P2 * duD + P5 * c1;
    const double a22 = P1 * c2 * c2 + P2 * dDD + P3 + 2 * P5 * c2;
    add_quadratic(H, a11, a12, a22, G12[0], G12[1]);

    // coefficients of the scalar Hessians
    const double bu = P2 * c1;            // on H_u (PT/EE) or H_N (PE)
    const double bD = P2 * c2 + P4;       // on H_D (PT/EE) or H_e (PE)
    double M[4][9];
    if (type >= 2) {
        // H_D Gram part: 2 (dn)^T(dn), dn/dX_i = alpha_i(-[B]x) + beta_i [A]x
        for (int i = 0; i < 4; i++) {
            double* Mi = M[i];
            double sa = al[i], sb = be[i];
            // -[B]x * sa + [A]x * sb
            double v0 = -sa * B[0] + sb * A[0], v1 = -sa * B[1] + sb * A[1], v2 = -sa * B[2] + sb * A[2];
            Mi[0] = 0; Mi[1] = -v2; Mi[2] = v1;
            Mi[3] = v2; Mi[4] = 0; Mi[5] = -v0;
            Mi[6] = -v1; Mi[7] = v0; Mi[8] = 0;
        }
        add_gram(H, 2 * bD, V, lbody, 4, M);
        // skew pair blocks: s_ij = bu * s_ij(u) + bD * s_ij(D)
        for (int i = 0; i < 4; i++)
            for (int j = i + 1; j < 4; j++) {
                double sv[3];
                for (int k = 0; k < 3; k++) {
                    double su = -al[i] * be[j] * W[k] + al[j] * be[i] * W[k]
                        + al[i] * ga[j] * B[k] - al[j] * ga[i] * B[k]
                        - be[i] * ga[j] * A[k] + be[j] * ga[i] * A[k];
                    double sD = 2 * (-al[i] * be[j] * n[k] + al[j] * be[i] * n[k]);
                    sv[k] = bu * su + bD * sD;
                }
                if (sv[0] == 0 && sv[1] == 0 && sv[2] == 0) continue;
                add_skew_pair(H, V[i], lbody[i], V[j], lbody[j], sv);
            }
    } else if (type == 1) {
        // H_N = 2 (dc)^T(dc) + skew(c); H_e = 2 (de)^T(de)
        for (int i = 0; i < 3; i++) {
            double* Mi = M[i];
            double sa = al[i], sb = be[i];
            double v0 = -sa * B[0] + sb * A[0], v1 = -sa * B[1] + sb * A[1], v2 = -sa * B[2] + sb * A[2];
            Mi[0] = 0; Mi[1] = -v2; Mi[2] = v1;
            Mi[3] = v2; Mi[4] = 0; Mi[5] = -v0;
            Mi[6] = -v1; Mi[7] = v0; Mi[8] = 0;
        }
        add_gram(H, 2 * bu, V, lbody, 3, M);
        for (int i = 0; i < 3; i++) {
            double* Mi = M[i];
            for (int k = 0; k < 9; k++) Mi[k] = 0;
            Mi[0] = Mi[4] = Mi[8] = ga[i];
        }
        add_gram(H, 2 * bD, V, lbody, 3, M);
        for (int i = 0; i < 3; i++)
            for (int j = i + 1; j < 3; j++) {
                double sv[3];
                for (int k = 0; k < 3; k++)
                    sv[k] = bu * 2 * (-al[i] * be[j] * n[k] + al[j] * be[i] * n[k]);
                if (sv[0] == 0 && sv[1] == 0 && sv[2] == 0) continue;
                add_skew_pair(H, V[i], lbody[i], V[j], lbody[j], sv);
            }
    } else {
        // d = |w|^2: hess = 2 (dw)^T (dw), coefficient P2 (c1 = 1)
        for (int i = 0; i < 2; i++) {
            double* Mi = M[i];
            for (int k = 0; k < 9; k++) Mi[k] = 0;
            Mi[0] = Mi[4] = Mi[8] = ga[i];
        }
        add_gram(H, 2 * P2, V, lbody, 2, M);
    }
    // curvature of the rigid maps
    add_curvature(H, fr, lbody, nvc, vrest, gv);
    return true;
}


template <int W>
__global__ void __launch_bounds__(kBarrierTPB) k_barrier_local(BarrierArgs a, int per_warp)
{
    extern __shared__ double smem[];
    local_terms<W>(a.n, per_warp, a.flags, a.hess, a.blocks, smem,
                   [&](int64_t ci, SMat H) { return barrier_build(a, ci, H); });
}

size_t local_terms_smem_bytes(int per_warp)
{
    return (size_t)(kRed * kRed) * (per_warp | 1) * sizeof(double);
}

// Constraints per warp: a thread per constraint (32) once they give every SM
// eight warps, fewer for small sets, down to 2 (16 lanes to each).  A power of
// two; tuned > 0: at most that.
int local_terms_per_warp(int64_t n, int tuned)
{
    const int64_t w = tuned > 0 ? tuned : (n + kNumSMs * 8 - 1) / (kNumSMs * 8);
    int p = 2;
    while (p < kBarrierTPB && p < w) p *= 2;
    return p;
}

static int launch_barrier(const BarrierArgs& a, int per_warp, cudaStream_t st)
{
    const unsigned grid = grid_for(a.n, per_warp);
    const size_t smem = local_terms_smem_bytes(per_warp);
    RIGC_COUNT_LAUNCH();
    switch (per_warp) {
    case 2: k_barrier_local<16><<<grid, kBarrierTPB, smem, st>>>(a, per_warp); break;
    case 4: k_barrier_local<8><<<grid, kBarrierTPB, smem, st>>>(a, per_warp); break;
    case 8: k_barrier_local<4><<<grid, kBarrierTPB, smem, st>>>(a, per_warp); break;
    case 16: k_barrier_local<2><<<grid, kBarrierTPB, smem, st>>>(a, per_warp); break;
    default: k_barrier_local<1><<<grid, kBarrierTPB, smem, st>>>(a, per_warp);
    }
    RIGC_CUDA(cudaGetLastError());
    return RIGC_OK;
}

int launch_body_frames(Ctx& c, const double* x)
{
    RIGC_TRY(c.frames.reserve((size_t)c.s.nb * 96 * sizeof(double)));
    RIGC_COUNT_LAUNCH();
    k_body_frames<<<grid_for(c.s.nb, 128), 128, 0, c.stream>>>(x, c.s.nb, c.frames.as<double>());
    RIGC_CUDA(cudaGetLastError());
    return RIGC_OK;
}

int launch_barrier_local(Ctx& c, const double* x, double dhat, double dmin, int flags,
                         double* energy, double* grad, double* blocks, double* hess)
{
    RIGC_TRY(launch_body_frames(c, x));
    if (c.cons.num == 0) return RIGC_OK;
    BarrierArgs a;
    a.rest = c.s.rest;
    a.frames = c.frames.as<double>();
    a.ctype = c.cons.type.as<int>();
    a.cverts = c.cons.verts.as<int>();
    a.cbodies = c.cons.bodies.as<int>();
    a.cweight = c.cons.weight.as<double>();
    a.ceps = c.cons.eps.as<double>();
    a.n = c.cons.num;
    a.dhat = dhat;
    a.dmin = dmin;
    a.flags = flags;
    a.energy = energy;
    a.grad = grad;
    a.blocks = blocks;
    a.hess = hess;
    return launch_barrier(a, local_terms_per_warp(c.cons.num, c.tune.barrier_per_warp), c.stream);
}

// Frames and per-constraint terms with every buffer supplied by the caller
// (the frames array holds 96 doubles per body); used by the entry point that
// allocates nothing.
int launch_barrier_local_raw(const double* rest, int64_t nv, int nb, const double* x, int64_t n,
                             const int* ctype, const int* cverts, const int* cbodies,
                             const double* cweight, const double* ceps, double dhat, double dmin,
                             int flags, double* frames, double* energy, double* grad,
                             double* hess, cudaStream_t stream)
{
    RIGC_COUNT_LAUNCH();
    k_body_frames<<<grid_for(nb, 128), 128, 0, stream>>>(x, nb, frames);
    RIGC_CUDA(cudaGetLastError());
    if (n == 0) return RIGC_OK;
    BarrierArgs a;
    a.rest = rest;
    a.frames = frames;
    a.ctype = ctype;
    a.cverts = cverts;
    a.cbodies = cbodies;
    a.cweight = cweight;
    a.ceps = ceps;
    a.n = n;
    a.dhat = dhat;
    a.dmin = dmin;
    a.flags = flags;
    a.energy = energy;
    a.grad = grad;
    a.blocks = nullptr;
    a.hess = hess;
    a.check_nb = nb;
    a.check_nv = nv;
    return launch_barrier(a, local_terms_per_warp(n, 0), stream);
}

// ---------------------------------------------------------------------------
// deterministic assembly: sort block keys, sum equal keys in constraint order

__global__ void k_block_keys(const int* __restrict__ bodies, int64_t n, int nb,
                             uint64_t* __restrict__ keys, uint32_t* __restrict__ vals)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 4 * n) return;
    int64_t c = i >> 2;
    int blk = (int)(i & 3);
    int bi = bodies[2 * c + (blk >> 1)], bj = bodies[2 * c + (blk & 1)];
    keys[i] = (uint64_t)bi * (uint64_t)nb + (uint64_t)bj;
    vals[i] = (uint32_t)i;
}

__global__ void k_grad_keys(const int* __restrict__ bodies, int64_t n,
                            uint32_t* __restrict__ keys, uint32_t* __restrict__ vals)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * n) return;
    keys[i] = (uint32_t)bodies[i];
    vals[i] = (uint32_t)i;
}

template <class Key>
__global__ void k_heads(const Key* __restrict__ keys, int64_t m, int32_t* __restrict__ head)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    head[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

// segment starts: seg_start[segid] = i for heads
__global__ void k_seg_starts(const int32_t* __restrict__ head, const int32_t* __restrict__ segid,
                             int64_t m, int32_t* __restrict__ seg_start)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    if (head[i]) seg_start[segid[i]] = (int32_t)i;
}

// the segment `seg` of key k, after one of key `before` (seg > 0): its
// column, and the row pointers between the two rows
__device__ __forceinline__ void block_segment(uint64_t k, uint64_t before, int32_t seg, int64_t start, int nb,
                                              int32_t* __restrict__ seg_start, int32_t* __restrict__ col,
                                              int32_t* __restrict__ row_ptr)
{
    seg_start[seg] = (int32_t)start;
    const int32_t r = (int32_t)(k / (uint64_t)nb);
    col[seg] = (int32_t)(k - (uint64_t)r * (uint64_t)nb);
    for (int32_t q = seg ? (int32_t)(before / (uint64_t)nb) + 1 : 0; q <= r; q++) row_ptr[q] = seg;
}

// the same for the sorted Hessian block keys, with columns and row pointers
__global__ void k_block_segs(const uint64_t* __restrict__ keys, const int32_t* __restrict__ head,
                             const int32_t* __restrict__ segid, int64_t m, int nb,
                             int32_t* __restrict__ seg_start, int32_t* __restrict__ col,
                             int32_t* __restrict__ row_ptr)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    if (head[i]) block_segment(keys[i], i ? keys[i - 1] : 0, segid[i], i, nb, seg_start, col, row_ptr);
    if (i == m - 1)
        for (int32_t q = (int32_t)(keys[i] / (uint64_t)nb) + 1; q <= nb; q++) row_ptr[q] = segid[i] + head[i];
}

// Few blocks: the sort of the keys by rank (the number of smaller keys, or
// equal ones before; keys from the constraints' bodies as k_block_keys has
// them), then the segments by one block; *nseg: their number.
constexpr int kRankBlocks = 4096;

__global__ void __launch_bounds__(128) k_rank_blocks(const int* __restrict__ bodies, int m, int nb,
                                                     uint64_t* __restrict__ out, uint32_t* __restrict__ slots)
{
    __shared__ uint64_t sh[1024];
    const auto key = [&](int i) {
        const int c = i >> 2, blk = i & 3;
        return (uint64_t)bodies[2 * c + (blk >> 1)] * (uint64_t)nb + (uint64_t)bodies[2 * c + (blk & 1)];
    };
    const int i = blockIdx.x * 128 + threadIdx.x;
    const uint64_t k = i < m ? key(i) : 0;
    int rank = 0;
    for (int c = 0; c < m; c += 1024) {
        const int n = min(1024, m - c);
        for (int j = threadIdx.x; j < n; j += 128) sh[j] = key(c + j);
        __syncthreads();
        for (int j = 0; j < n; j++) rank += sh[j] < k || (sh[j] == k && c + j < i);
        __syncthreads();
    }
    if (i >= m) return;
    out[rank] = k;
    slots[rank] = (uint32_t)i;
}

__global__ void __launch_bounds__(1024) k_block_segs_small(const uint64_t* __restrict__ keys, int m, int nb,
                                                           int32_t* __restrict__ seg_start, int32_t* __restrict__ col,
                                                           int32_t* __restrict__ row_ptr, int32_t* __restrict__ nseg)
{
    __shared__ int32_t warp_sum[32];
    __shared__ int32_t carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < m; base += 1024) {
        const int i = base + (int)threadIdx.x;
        const bool head = i < m && (i == 0 || keys[i] != keys[i - 1]);
        const unsigned b = __ballot_sync(0xffffffffu, head);
        if (lane == 0) warp_sum[warp] = __popc(b);
        __syncthreads();
        int s = carry;
        for (int w = 0; w < warp; w++) s += warp_sum[w];
        s += __popc(b & ((1u << lane) - 1u));
        if (head) block_segment(keys[i], i ? keys[i - 1] : 0, s, i, nb, seg_start, col, row_ptr);
        __syncthreads();
        if (threadIdx.x == 1023) carry = s + (head ? 1 : 0);
        __syncthreads();
    }
    const int total = carry;
    for (int32_t q = (int32_t)(keys[m - 1] / (uint64_t)nb) + 1 + (int)threadIdx.x; q <= nb; q += 1024) row_ptr[q] = total;
    if (threadIdx.x == 0) *nseg = total;
}

// Sum of a segment's items by a block, one thread per (slice, entry): slice s
// takes items s, s + S, ... in order, then the slices are added in order, so
// the sum depends on the segment's items alone and one of at most S items is
// the sequential sum.  A few bodies in face-to-face contact give segments of
// 10^4 items (172 k constraints between 33 bodies: one thread per entry took
// 4.3 ms for the blocks and 2.4 ms for the gradient, the latency of a chain of
// adds; the slices take 0.22 and 0.1 ms).
template <int E, int S, class Load>
__device__ __forceinline__ double segment_sum(int64_t s0, int64_t s1, double* part, Load load)
{
    const int e = threadIdx.x % E, s = threadIdx.x / E;
    double acc = 0;
    int64_t i = s < S ? s0 + s : s1;
    for (; i + 3 * S < s1; i += 4 * S) {
        const double a = load(i, e), b = load(i + S, e), c = load(i + 2 * S, e), d = load(i + 3 * S, e);
        acc = (((acc + a) + b) + c) + d;
    }
    for (; i < s1; i += S) acc += load(i, e);
    if (s < S) part[s * E + e] = acc;
    __syncthreads();
    double sum = 0;
    if (s == 0) {
        const int64_t used = s1 - s0 < S ? s1 - s0 : S;
        for (int k = 0; k < used; k++) sum += part[k * E + e];
    }
    __syncthreads();
    return sum;
}

constexpr int kBlockSlices = 16, kGradSlices = 64;

// Blocks over the unique Hessian blocks.  A diagonal block's segment lists
// its body's constraints (slot 4 c: its first body, 4 c + 3: its second) in the
// order of the gradient's own segment, so its block sums the body's gradient
// too.
__global__ void __launch_bounds__(36 * kBlockSlices) k_block_sums(
    const uint64_t* __restrict__ keys, const uint32_t* __restrict__ slots, const int32_t* __restrict__ seg_start,
    const int32_t* __restrict__ nseg_ptr, int64_t m, const double* __restrict__ blocks,
    const double* __restrict__ cgrad, int nb, double* __restrict__ val, double* __restrict__ grad)
{
    __shared__ double part[36 * kBlockSlices];
    const int32_t nseg = *nseg_ptr;
    for (int32_t sgi = blockIdx.x; sgi < nseg; sgi += gridDim.x) {
        const int64_t s0 = seg_start[sgi], s1 = sgi + 1 < nseg ? seg_start[sgi + 1] : m;
        const double sum = segment_sum<36, kBlockSlices>(
            s0, s1, part, [&](int64_t i, int e) { return blocks[(size_t)slots[i] * 36 + e]; });
        if (threadIdx.x < 36) val[(size_t)sgi * 36 + threadIdx.x] = sum;
        const uint64_t k = keys[s0];
        const uint32_t row = (uint32_t)(k / (uint64_t)nb);
        if (k != (uint64_t)row * (uint64_t)nb + row) continue;  // uniform over the block
        const double g = segment_sum<6, kGradSlices>(s0, s1, part, [&](int64_t i, int e) {
            const uint32_t slot = slots[i];
            return cgrad[(size_t)(slot >> 2) * 12 + 6 * ((slot & 3) == 3) + e];
        });
        if (threadIdx.x < 6) grad[(size_t)row * 6 + threadIdx.x] = g;
    }
}

// blocks over the bodies with a gradient
__global__ void __launch_bounds__(6 * kGradSlices) k_grad_sums(
    const uint32_t* __restrict__ keys, const uint32_t* __restrict__ slots, const int32_t* __restrict__ seg_start,
    const int32_t* __restrict__ nseg_ptr, int64_t m, const double* __restrict__ cgrad, double* __restrict__ grad)
{
    __shared__ double part[6 * kGradSlices];
    const int32_t nseg = *nseg_ptr;
    for (int32_t sgi = blockIdx.x; sgi < nseg; sgi += gridDim.x) {
        const int64_t s0 = seg_start[sgi], s1 = sgi + 1 < nseg ? seg_start[sgi + 1] : m;
        const double sum = segment_sum<6, kGradSlices>(s0, s1, part, [&](int64_t i, int e) {
            const uint32_t slot = slots[i];  // = 2 c + side
            return cgrad[(size_t)(slot >> 1) * 12 + 6 * (slot & 1) + e];
        });
        if (threadIdx.x < 6) grad[(size_t)keys[s0] * 6 + threadIdx.x] = sum;
    }
}

int assemble_terms(Ctx& c, const int* bodies, int64_t n, const double* cgrad,
                   const double* cblocks, DevBuf& grad, DevBuf& row_ptr, DevBuf& col,
                   DevBuf& val, int32_t* nseg_dev_pair, bool with_hess)
{
    const int nb = c.s.nb;
    cudaStream_t st = c.stream;
    RIGC_TRY(grad.reserve((size_t)6 * nb * sizeof(double)));
    RIGC_TRY(row_ptr.reserve((size_t)(nb + 1) * sizeof(int32_t)));
    RIGC_CUDA(cudaMemsetAsync(grad.ptr, 0, (size_t)6 * nb * sizeof(double), st));
    RIGC_CUDA(cudaMemsetAsync(row_ptr.ptr, 0, (size_t)(nb + 1) * sizeof(int32_t), st));
    if (n == 0) return RIGC_OK;
    // scratch usage: 0 keys_in, 1 vals_in, 2 keys_out, 3 vals_out, 4/5 sort tmp,
    // 6 hist/scan tmp, 7 head/segid/seg_start
    DevBuf* S = c.scratch;
    if (!with_hess) {
        // the gradient alone, by body
        int64_t m = 2 * n;
        RIGC_TRY(S[0].reserve(m * 4));
        RIGC_TRY(S[1].reserve(m * 4));
        RIGC_TRY(S[2].reserve(m * 4));
        RIGC_TRY(S[3].reserve(m * 4));
        RIGC_TRY(S[7].reserve(m * 12 + 16));
        RIGC_COUNT_LAUNCH();
        k_grad_keys<<<grid_for(m, 256), 256, 0, st>>>(bodies, n, S[0].as<uint32_t>(),
                                                     S[1].as<uint32_t>());
        RIGC_TRY(radix_sort_pairs<uint32_t>(S[0].as<uint32_t>(), S[1].as<uint32_t>(),
                                            S[2].as<uint32_t>(), S[3].as<uint32_t>(), m,
                                            bits_for((uint64_t)nb), S[4], S[5], S[6], st));
        int32_t* head = S[7].as<int32_t>();
        int32_t* segid = head + m;
        int32_t* segst = segid + m;
        RIGC_COUNT_LAUNCH();
        k_heads<uint32_t><<<grid_for(m, 256), 256, 0, st>>>(S[2].as<uint32_t>(), m, head);
        int32_t* nseg_dev = nseg_dev_pair;
        RIGC_TRY(exclusive_scan_i32(head, segid, m, nseg_dev, S[6], st));
        RIGC_COUNT_LAUNCH();
        k_seg_starts<<<grid_for(m, 256), 256, 0, st>>>(head, segid, m, segst);
        // at most m segments; the kernel reads the true count on the device
        RIGC_COUNT_LAUNCH();
        k_grad_sums<<<(unsigned)std::min<int64_t>(m, kNumSMs * 4), 6 * kGradSlices, 0, st>>>(
            S[2].as<uint32_t>(), S[3].as<uint32_t>(), segst, nseg_dev, m, cgrad,
            grad.as<double>());
        return RIGC_OK;
    }
    const int64_t m = 4 * n;
    RIGC_TRY(S[2].reserve(m * 8));
    RIGC_TRY(S[3].reserve(m * 4));
    RIGC_TRY(S[7].reserve(m * 12 + 16));
    // capacity for the upper bound m blocks: no host round trip here
    RIGC_TRY(col.reserve((size_t)m * sizeof(int32_t)));
    RIGC_TRY(val.reserve((size_t)m * 36 * sizeof(double)));
    int32_t* head = S[7].as<int32_t>();
    int32_t* segid = head + m;
    int32_t* segst = segid + m;
    int32_t* nseg_dev = nseg_dev_pair + 1;  // read back by the caller
    if (m <= kRankBlocks) {
        RIGC_COUNT_LAUNCH();
        k_rank_blocks<<<grid_for(m, 128), 128, 0, st>>>(bodies, (int)m, nb, S[2].as<uint64_t>(),
                                                        S[3].as<uint32_t>());
        RIGC_COUNT_LAUNCH();
        k_block_segs_small<<<1, 1024, 0, st>>>(S[2].as<uint64_t>(), (int)m, nb, segst, col.as<int32_t>(),
                                               row_ptr.as<int32_t>(), nseg_dev);
    } else {
        RIGC_TRY(S[0].reserve(m * 8));
        RIGC_TRY(S[1].reserve(m * 4));
        RIGC_COUNT_LAUNCH();
        k_block_keys<<<grid_for(m, 256), 256, 0, st>>>(bodies, n, nb,
                                                      S[0].as<uint64_t>(), S[1].as<uint32_t>());
        RIGC_TRY(radix_sort_pairs<uint64_t>(S[0].as<uint64_t>(), S[1].as<uint32_t>(),
                                            S[2].as<uint64_t>(), S[3].as<uint32_t>(), m,
                                            bits_for((uint64_t)nb * nb), S[4], S[5], S[6], st));
        RIGC_COUNT_LAUNCH();
        k_heads<uint64_t><<<grid_for(m, 256), 256, 0, st>>>(S[2].as<uint64_t>(), m, head);
        RIGC_TRY(exclusive_scan_i32(head, segid, m, nseg_dev, S[6], st));
        RIGC_COUNT_LAUNCH();
        k_block_segs<<<grid_for(m, 256), 256, 0, st>>>(S[2].as<uint64_t>(), head, segid, m, nb, segst,
                                                       col.as<int32_t>(), row_ptr.as<int32_t>());
    }
    RIGC_COUNT_LAUNCH();
    k_block_sums<<<(unsigned)std::min<int64_t>(m, kNumSMs * 3), 36 * kBlockSlices, 0, st>>>(
        S[2].as<uint64_t>(), S[3].as<uint32_t>(), segst, nseg_dev, m, cblocks, cgrad, nb, val.as<double>(),
        grad.as<double>());
    RIGC_CUDA(cudaGetLastError());
    return RIGC_OK;
}

// Per-scene sums of per-constraint values in constraint order.  Within each
// type segment the constraints are ordered by their first primitive, hence
// by body and by scene; each thread binary-searches its scene's range in the
// four segments.
__global__ void k_scene_sums(const double* __restrict__ val, const int* __restrict__ bodies,
                             const int* __restrict__ bscene, int4 seg_start, int64_t n,
                             int nscenes, double* __restrict__ out)
{
    int sc = blockIdx.x * blockDim.x + threadIdx.x;
    if (sc >= nscenes) return;
    const int64_t starts[5] = { seg_start.x, seg_start.y, seg_start.z, seg_start.w, n };
    double acc = 0;
    for (int t = 0; t < 4; t++) {
        int64_t lo = starts[t], hi = starts[t + 1];
        // first constraint of the segment with scene >= sc
        int64_t a = lo, b = hi;
        while (a < b) {
            int64_t m = (a + b) / 2;
            if (bscene[bodies[2 * m]] < sc) a = m + 1;
            else b = m;
        }
        for (int64_t i = a; i < hi && bscene[bodies[2 * i]] == sc; i++) acc += val[i];
    }
    out[sc] = acc;
}

int scene_sums(Ctx& c, const double* val, const int* bodies, int64_t n, const int64_t seg[4],
               std::vector<double>& out)
{
    const int ns = c.s.nscenes;
    out.assign(ns, 0.0);
    if (n == 0) return RIGC_OK;
    RIGC_TRY(c.scene_energy.reserve((size_t)ns * 8 + 8));
    int4 st4 = make_int4((int)seg[0], (int)seg[1], (int)seg[2], (int)seg[3]);
    RIGC_COUNT_LAUNCH();
    k_scene_sums<<<grid_for(ns, 128), 128, 0, c.stream>>>(val, bodies, c.s.bscene, st4, n, ns,
                                                          c.scene_energy.as<double>());
    RIGC_CUDA(cudaMemcpyAsync(out.data(), c.scene_energy.ptr, (size_t)ns * 8, cudaMemcpyDeviceToHost,
                              c.stream));
    RIGC_CUDA(cudaStreamSynchronize(c.stream));
    return RIGC_OK;
}

int assemble_barrier(Ctx& c, bool with_hess)
{
    // on the device (d_scalars int 1) until the caller syncs
    c.nnzb = (with_hess && c.cons.num > 0) ? -1 : 0;
    return assemble_terms(c, c.cons.bodies.as<int>(), c.cons.num, c.c_grad.as<double>(),
                          c.c_blocks.as<double>(), c.grad, c.row_ptr, c.col, c.val,
                          c.d_scalars.as<int32_t>(), with_hess);
}

} // namespace rigc

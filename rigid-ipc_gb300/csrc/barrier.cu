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
// Derivation used by k_barrier_local.  The distances are functions of a few
// signed sums of the vertices:
//  * PT / EE: d = u^2 / D with u = n.W, n = A x B and D = |n|^2;
//  * PE: d = |n|^2 / |W|^2, W the edge;
//  * PP: d = |W|^2;
//  * a mollified EE whose closest feature is an endpoint has its edges' n and a
//    PE or PP distance of its own (P x Q and W).
// f = weight * m(D) * b(d - dmin^2) (m = 1 except mollified EE).  Along a pose
// coordinate the vectors move by dA .. dW (a body's part of A moves by dR/dtheta_k
// times that part's rest vector), which gives the scalars' derivatives; the body
// Hessian is a quadratic form of those, products of the moved vectors, and the
// curvature term sum_i grad_Xi f . d2X_i/dtheta2 (BarrierBase).  It is then
// projected to the PSD cone, V max(L, 0) V^T (local_terms.cuh).
#include <algorithm>

#include "common.cuh"
#include "geometry_rn.cuh"
#include "local_terms.cuh"
#include "rotation.cuh"
#include "sort.cuh"

namespace rigc {

// ---------------------------------------------------------------------------
// per-body frames (R, dR, d2R) and positions

// a warp per body, or (many bodies) a thread
template <bool kWarp>
__global__ void k_body_frames(const double* __restrict__ x, int nb, double* __restrict__ frames)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = kWarp ? i >> 5 : i;
    if (b >= nb) return;
    const double t[3] = { x[6 * b + 3], x[6 * b + 4], x[6 * b + 5] };
    double* out = frames + (size_t)b * 96;
    if (kWarp) {
        const int lane = threadIdx.x & 31;
        warp_body_frame(t, lane, out);
        if (lane < 3) out[90 + lane] = x[6 * b + lane];
        return;
    }
    double F[kFrameDoubles];
    body_frame(t, F);
#pragma unroll
    for (int k = 0; k < kFrameDoubles; k++) out[k] = F[k];
    for (int k = 0; k < 3; k++) out[90 + k] = x[6 * b + k];
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

// What a constraint's terms are made of: cross products n = A x B and c = P x Q
// (c: the point-edge distance of a mollified EE whose closest feature is an
// endpoint) and a vector W, each of A, B, P, Q, W a signed sum of the vertices.
// Along coordinate r of the bodies' poses they move by dA .. dW, and with
//   N' = tn.dn + tw.dW + tc.dc,  E' = 2 W.dW,  D' = 2 n.dn
// the gradient is g.(N', E', D') and the Hessian entry
//   (N', E', D') C (N', E', D')^T + k1 dn.dn + kx (dn.dW + dW.dn) + kw dW.dW
//   + k2 dc.dc + y1 (dA x dB + dA x dB) n + y2 (dP x dQ + dP x dQ) c (W's part
//   of the vector in Y1), the products of coordinate r's and column's vectors,
// plus the curvature of the rotations, the second derivatives of the vertices.
struct BarrierBase {
    double A[3], B[3], P[3], Q[3], W[3];
    double n[3], c[3];
    double tn[3], tw[3], tc[3];
    double Y1[3], Y2[3];
    double k1, kx, kw, k2;
    double C[6];              // NN, NE, ND, EE, ED, DD
    double g[3];
    double f[5][3];           // derivatives of f in A .. W
    double s[5];              // sums of A, B, P, Q, W's coefficients on body a's vertices
    double v[2][5][3];        // the bodies' parts of A .. W in rest positions
    double S[2][9];           // sum of (df/dX_i) v_i^T over the bodies' vertices
    int cross2;               // P, Q, c are there
};
constexpr int kCoord = 24;    // stored per coordinate: Y1 x dA, dB, dn, dW, N', E', D', Y2 x dP, dQ, dc
enum BarrierState { kNothing, kGradient, kHessian };

__device__ __forceinline__ void add_outer3(double* S, const double* g, const double* v)
{
    for (int j = 0; j < 3; j++)
        for (int k = 0; k < 3; k++) S[3 * j + k] = fma(g[j], v[k], S[3 * j + k]);
}

// The vectors, scalars and coefficients of a constraint; its energy.  Run by
// every lane of the constraint's group, written by the first.
static __device__ __noinline__ int barrier_base(const BarrierArgs& a, int64_t ci, bool first, BarrierBase& o)
{
    auto fill = [&](double v) {
        if (!first) return;
        if (a.grad)
            for (int k = 0; k < 12; k++) a.grad[ci * 12 + k] = v;
        if (a.flags & RIGC_HESS) {
            if (a.blocks)
                for (int k = 0; k < 144; k++) a.blocks[ci * 144 + k] = v;
            if (a.hess)
                for (int k = 0; k < 144; k++) a.hess[ci * 144 + k] = v;
        }
    };
    if (a.check_nv >= 0 && !constraint_in_range(a, ci)) {
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        if (a.energy && first) a.energy[ci] = nan;
        fill(nan);
        return kNothing;
    }
    const int type = a.ctype[ci];
    const int nvc = type == 0 ? 2 : (type == 1 ? 3 : 4);
    const double weight = a.cweight[ci];
    double X[4][3], vr[4][3];
    for (int i = 0; i < nvc; i++) {
        const double* f = a.frames + (size_t)a.cbodies[2 * ci + local_body_of(type, i)] * 96;
        const int vi = a.cverts[4 * ci + i];
        for (int j = 0; j < 3; j++) vr[i][j] = a.rest[3 * (size_t)vi + j];
        for (int j = 0; j < 3; j++)
            X[i][j] = f[3 * j] * vr[i][0] + f[3 * j + 1] * vr[i][1] + f[3 * j + 2] * vr[i][2] + f[90 + j];
    }
    // end: an EE's closest feature is an endpoint: 1 two points, 2 a point and an edge
    int end = 0, p = 0, e0 = 0, e1 = 0;
    if (type == 2) {
        switch (ee_type_rn(X[0], X[1], X[2], X[3])) {
        case EE_EA_EB: break;
        case EE_EA0_EB0: end = 1; p = 0; e0 = 2; break;
        case EE_EA0_EB1: end = 1; p = 0; e0 = 3; break;
        case EE_EA1_EB0: end = 1; p = 1; e0 = 2; break;
        case EE_EA1_EB1: end = 1; p = 1; e0 = 3; break;
        case EE_EA_EB0: end = 2; p = 2; e0 = 0; e1 = 1; break;
        case EE_EA_EB1: end = 2; p = 3; e0 = 0; e1 = 1; break;
        case EE_EA0_EB: end = 2; p = 0; e0 = 2; e1 = 3; break;
        default: end = 2; p = 1; e0 = 2; e1 = 3; break;
        }
    }
    // the vectors as differences of vertices (to, from)
    int to[5] = { 0, 0, 0, 0, 0 }, from[5] = { 0, 0, 0, 0, 0 };
    if (type == 2) {        // A = X1 - X0, B = X3 - X2, W = X2 - X0
        to[0] = 1; to[1] = 3; from[1] = 2; to[4] = 2;
        if (end == 1) {     // W between the two points
            to[4] = p; from[4] = e0;
        } else if (end == 2) {  // P, Q from the point to the edge's ends, W the edge
            to[2] = e0; from[2] = p; to[3] = e1; from[3] = p; to[4] = e1; from[4] = e0;
        }
    } else if (type == 3) { // A = X2 - X1, B = X3 - X1, W = X0 - X1
        to[0] = 2; from[0] = 1; to[1] = 3; from[1] = 1; from[4] = 1;
    } else if (type == 1) { // A = X1 - X0, B = X2 - X0, W the edge X2 - X1
        to[0] = 1; to[1] = 2; to[4] = 2; from[4] = 1;
    } else {                // W = X0 - X1
        from[4] = 1;
    }
    o.cross2 = end == 2;
    double* vec[5] = { o.A, o.B, o.P, o.Q, o.W };
    for (int q = 0; q < 5; q++) {
        const int t = to[q], f = from[q], bt = local_body_of(type, t), bf = local_body_of(type, f);
        for (int j = 0; j < 3; j++) {
            vec[q][j] = X[t][j] - X[f][j];
            const double vt = vr[t][j], vf = vr[f][j];
            o.v[0][q][j] = (bt == 0 ? vt : 0.0) - (bf == 0 ? vf : 0.0);
            o.v[1][q][j] = (bt == 1 ? vt : 0.0) - (bf == 1 ? vf : 0.0);
        }
        o.s[q] = (double)((bt == 0) - (bf == 0));
    }
    cross(o.A, o.B, o.n);
    cross(o.P, o.Q, o.c);
    const double nn = dot(o.n, o.n), ww = dot(o.W, o.W), cc = dot(o.c, o.c);
    double u = 0, d;
    if (type == 0 || end == 1) {
        d = ww;
    } else if (type == 1) {
        d = nn / ww;
    } else if (end == 2) {
        d = cc / ww;
    } else {
        u = dot(o.n, o.W);
        d = u * u / nn;
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
    if (type == 2 && nn < a.ceps[ci]) {
        double ie = 1.0 / a.ceps[ci];
        double xe = nn * ie;
        m = (2 - xe) * xe;
        m1 = (2 - 2 * xe) * ie;
        m2 = -2 * ie * ie;
    }
    if (a.energy && first) a.energy[ci] = weight * m * bv;
    if (!active) {
        fill(0.0);
        return kNothing;
    }
    if (!(a.flags & (RIGC_GRAD | RIGC_HESS))) return kNothing;

    // f = weight m(D) b(d).  Hessian of d in the scalars:
    //  PT/EE: (2/D) u'u' - (2u/D^2)(u'D' + D'u') + (2u^2/D^3) D'D' + (2u/D) u'' - (u^2/D^2) D''
    //  PE:    -(1/E^2)(N'E' + E'N') + (2N/E^3) E'E' + (1/E) N'' - (N/E^2) E'',  E = |W|^2
    //  PP:    W''
    const double wm = weight * m;
    const double P1 = wm * b2, P2 = wm * b1;               // on d'd' and d''
    const double P3 = weight * bv * m2, P4 = weight * bv * m1, P5 = weight * m1 * b1;  // D'D', D'', d'D' (EE)
    for (int q = 0; q < 6; q++) o.C[q] = 0;
    for (int j = 0; j < 3; j++) o.tn[j] = o.tw[j] = o.tc[j] = o.Y1[j] = o.Y2[j] = 0;
    o.k1 = o.kx = o.kw = o.k2 = 0;
    o.g[0] = o.g[1] = o.g[2] = 0;
    if (type == 0 || end == 1) {
        o.C[0] = P1;
        o.C[2] = P5;
        o.C[5] = P3;
        o.g[0] = P2;
        o.g[2] = P4;
        o.kw = 2 * P2;
        o.k1 = 2 * P4;
        for (int j = 0; j < 3; j++) {
            o.tw[j] = 2 * o.W[j];
            o.Y1[j] = 2 * P4 * o.n[j];
        }
    } else if (type == 1 || end == 2) {
        const double N = type == 1 ? nn : cc, c1 = 1 / ww, c2 = -N / (ww * ww);
        o.C[0] = P1 * c1 * c1;
        o.C[1] = P1 * c1 * c2 - P2 / (ww * ww);
        o.C[3] = P1 * c2 * c2 + P2 * (2 * N / (ww * ww * ww));
        o.C[2] = P5 * c1;
        o.C[4] = P5 * c2;
        o.C[5] = P3;
        o.g[0] = P2 * c1;
        o.g[1] = P2 * c2;
        o.g[2] = P4;
        o.kw = 2 * P2 * c2;
        const double kN = 2 * P2 * c1;
        if (type == 1) o.k1 = kN;
        else {
            o.k1 = 2 * P4;
            o.k2 = kN;
        }
        for (int j = 0; j < 3; j++) {
            (type == 1 ? o.tn : o.tc)[j] = 2 * (type == 1 ? o.n : o.c)[j];
            o.Y1[j] = o.k1 * o.n[j];
            o.Y2[j] = o.k2 * o.c[j];
        }
    } else {
        const double c1 = 2 * u / nn, c2 = -u * u / (nn * nn);
        o.C[0] = P1 * c1 * c1 + P2 * (2 / nn);
        o.C[2] = P1 * c1 * c2 - P2 * (2 * u / (nn * nn)) + P5 * c1;
        o.C[5] = P1 * c2 * c2 + P2 * (2 * u * u / (nn * nn * nn)) + P3 + 2 * P5 * c2;
        o.g[0] = P2 * c1;
        o.g[2] = P2 * c2 + P4;
        o.kx = P2 * c1;
        o.k1 = 2 * (P2 * c2 + P4);
        for (int j = 0; j < 3; j++) {
            o.tn[j] = o.W[j];
            o.tw[j] = o.n[j];
            o.Y1[j] = o.kx * o.W[j] + o.k1 * o.n[j];
        }
    }
    // derivatives of f in A .. W, then S
    double q1[3], q2[3], (*gr)[3] = o.f;
    for (int j = 0; j < 3; j++) {
        q1[j] = o.g[0] * o.tn[j] + 2 * o.g[2] * o.n[j];
        q2[j] = o.g[0] * o.tc[j];
        gr[4][j] = o.g[0] * o.tw[j] + 2 * o.g[1] * o.W[j];
    }
    cross(o.B, q1, gr[0]);
    cross(q1, o.A, gr[1]);
    cross(o.Q, q2, gr[2]);
    cross(q2, o.P, gr[3]);
    if (!(a.flags & RIGC_HESS)) return kGradient;
    for (int b = 0; b < 2; b++) {
        for (int k = 0; k < 9; k++) o.S[b][k] = 0;
        for (int q = 0; q < 5; q++)
            if (o.cross2 || q < 2 || q == 4) add_outer3(o.S[b], gr[q], o.v[b][q]);
    }
    return kHessian;
}

__device__ __forceinline__ void fcross(const double* x, const double* y, double* r)
{
    for (int j = 0; j < 3; j++) {
        const int k = (j + 1) % 3, l = (j + 2) % 3;
        r[j] = fma(x[k], y[l], -__dmul_rn(x[l], y[k]));
    }
}
__device__ __forceinline__ double fdot(const double* x, const double* y, double s)
{
    return fma(x[2], y[2], fma(x[1], y[1], fma(x[0], y[0], s)));
}

// Coordinate r: its vectors and scalars into st, its gradient
static __device__ __noinline__ double barrier_coord(const BarrierBase& o, const double* fa, const double* fb, int r,
                                                    double* st, int stride)
{
    double d[5][3];
    if (r < 3) {
        for (int q = 0; q < 5; q++)
            for (int j = 0; j < 3; j++) d[q][j] = j == r ? o.s[q] : 0.0;
    } else {
        const int b = r >= 6;
        const double* M = (b ? fb : fa) + 9 + 9 * (r - (b ? 6 : 3));
        for (int q = 0; q < 5; q++) {
            if ((q == 2 || q == 3) && !o.cross2) continue;
            for (int j = 0; j < 3; j++) d[q][j] = fdot(M + 3 * j, o.v[b][q], 0.0);
        }
    }
    double x[3], y[3], dn[3];
    fcross(d[0], o.B, x);
    fcross(o.A, d[1], y);
    for (int j = 0; j < 3; j++) dn[j] = __dadd_rn(x[j], y[j]);
    fcross(o.Y1, d[0], x);
    double N = fdot(o.tn, dn, fdot(o.tw, d[4], 0.0));
    for (int j = 0; j < 3; j++) {
        st[j * stride] = x[j];
        st[(3 + j) * stride] = d[1][j];
        st[(6 + j) * stride] = dn[j];
        st[(9 + j) * stride] = d[4][j];
    }
    if (o.cross2) {
        double dc[3];
        fcross(d[2], o.Q, x);
        fcross(o.P, d[3], y);
        for (int j = 0; j < 3; j++) dc[j] = __dadd_rn(x[j], y[j]);
        fcross(o.Y2, d[2], x);
        N = fdot(o.tc, dc, N);
        for (int j = 0; j < 3; j++) {
            st[(15 + j) * stride] = x[j];
            st[(18 + j) * stride] = d[3][j];
            st[(21 + j) * stride] = dc[j];
        }
    }
    const double E = __dmul_rn(2.0, fdot(o.W, d[4], 0.0)), D = __dmul_rn(2.0, fdot(o.n, dn, 0.0));
    st[12 * stride] = N;
    st[13 * stride] = E;
    st[14 * stride] = D;
    // by the forces on A .. W (the scalars' parts, N' and D' of a shallow angle
    // above all, cancel in them before they are rounded; by the scalars, in three
    // orders, the converged run of 27 landing cubes ends 1e-8 from the oracle's)
    double G = fdot(o.f[1], d[1], fdot(o.f[0], d[0], 0.0));
    if (o.cross2) G = fdot(o.f[3], d[3], fdot(o.f[2], d[2], G));
    return fdot(o.f[4], d[4], G);
}

// Entries (r, col), r <= col, from the coordinates' values
static __device__ __noinline__ void barrier_column(const BarrierBase& o, const double* fa, const double* fb, int col,
                                                   const double* st, int stride, SMat H)
{
    const double* sc = st + col * kCoord * stride;
    double ya[3], db[3], z[3], t[3], q[3];
    const double N = sc[12 * stride], E = sc[13 * stride], D = sc[14 * stride];
    q[0] = fma(o.C[2], D, fma(o.C[1], E, __dmul_rn(o.C[0], N)));
    q[1] = fma(o.C[4], D, fma(o.C[3], E, __dmul_rn(o.C[1], N)));
    q[2] = fma(o.C[5], D, fma(o.C[4], E, __dmul_rn(o.C[2], N)));
    for (int j = 0; j < 3; j++) {
        ya[j] = sc[j * stride];
        db[j] = sc[(3 + j) * stride];
        const double dn = sc[(6 + j) * stride], dw = sc[(9 + j) * stride];
        z[j] = fma(o.kx, dw, __dmul_rn(o.k1, dn));
        t[j] = fma(o.kw, dw, __dmul_rn(o.kx, dn));
    }
    for (int r = 0; r <= col; r++) {
        const double* sr = st + r * kCoord * stride;
        double h = fma(q[2], sr[14 * stride], fma(q[1], sr[13 * stride], __dmul_rn(q[0], sr[12 * stride])));
        double k = 0.0;
        for (int j = 0; j < 3; j++) {
            h = fma(sr[j * stride], db[j], h);
            k = fma(sr[(3 + j) * stride], ya[j], k);
            h = fma(sr[(6 + j) * stride], z[j], h);
            k = fma(sr[(9 + j) * stride], t[j], k);
        }
        H.at(r, col) = __dadd_rn(h, k);
    }
    if (o.cross2) {
        for (int j = 0; j < 3; j++) {
            ya[j] = sc[(15 + j) * stride];
            db[j] = sc[(18 + j) * stride];
            z[j] = __dmul_rn(o.k2, sc[(21 + j) * stride]);
        }
        for (int r = 0; r <= col; r++) {
            const double* sr = st + r * kCoord * stride;
            double h = H.at(r, col);
            for (int j = 0; j < 3; j++) {
                h = fma(sr[(15 + j) * stride], db[j], h);
                h = fma(sr[(18 + j) * stride], ya[j], h);
                h = fma(sr[(21 + j) * stride], z[j], h);
            }
            H.at(r, col) = h;
        }
    }
    if (col < 3) return;
    // curvature: the second derivatives of the column's body's rotation
    const int b = col >= 6, l = col - (b ? 6 : 3);
    const double* d2 = (b ? fb : fa) + 36;
    for (int k = 0; k <= l; k++) {
        const double* M = d2 + 9 * sym_index(k, l);
        double h = H.at(col - l + k, col);
        for (int e = 0; e < 9; e++) h = fma(M[e], o.S[b][e], h);
        H.at(col - l + k, col) = h;
    }
}

// The terms of a constraint by its group of W lanes, coordinates and columns
// dealt out to them.  Bound by FP64 issue: a warp instruction costs the same for
// 1 lane and for 32, so what the lanes share is worth its rate.  Every
// coordinate's values are few (Y1 x dA in place of dA: a pair's part of the
// second derivative is then two dot products), 15 to 24 multiply-adds an entry;
// by vertices (skew blocks J_i^T [s]x J_j, Gram terms of 3 x 9 Jacobians) one
// lane took some 2800 instructions.  Unprojected, with the frames: 338
// constraints of 27 cubes (16 lanes each) 210 -> 88 us, 163 k of 32 slabs (a lane
// each) 1.33 -> 0.85 ms.
template <int W>
__device__ __forceinline__ bool barrier_build(const BarrierArgs& a, int64_t ci, SMat H, int g, unsigned mask,
                                              double* scratch, int stride)
{
    BarrierBase o;
    const int state = barrier_base(a, ci, g == 0, o);
    if (state == kNothing) return false;
    double own[W == 1 ? kRed * kCoord : 1];
    double* st = W == 1 ? own : scratch;
    const int ss = W == 1 ? 1 : stride;
    const double* fa = a.frames + (size_t)a.cbodies[2 * ci] * 96;
    const double* fb = a.frames + (size_t)a.cbodies[2 * ci + 1] * 96;
    for (int r = g; r < kRed; r += W) {
        const double G = barrier_coord(o, fa, fb, r, st + r * kCoord * ss, ss);
        if (a.grad) {
            a.grad[ci * 12 + (r < 6 ? r : r + 3)] = G;
            if (r < 3) a.grad[ci * 12 + 6 + r] = -G;
        }
    }
    if (state != kHessian) return false;
    group_sync<W>(mask);
    // (from the last: the longest columns first)
    for (int c = kRed - 1 - g; c >= 0; c -= W) barrier_column(o, fa, fb, c, st, ss, H);
    return true;
}

template <int W>
__global__ void __launch_bounds__(kBarrierTPB) k_barrier_local(BarrierArgs a, int per_warp)
{
    extern __shared__ double smem[];
    const int stride = per_warp | 1;
    local_terms<W>(a.n, per_warp, a.flags, a.hess, a.blocks, smem, [&](int64_t ci, SMat H, int g, unsigned mask) {
        return barrier_build<W>(a, ci, H, g, mask, H.base + kRed * kRed * stride, stride);
    });
}

size_t local_terms_smem_bytes(int per_warp)
{
    return (size_t)(kRed * kRed) * (per_warp | 1) * sizeof(double);
}

// Constraints per warp: a thread per constraint (32) once they give every SM
// eight warps, fewer for small sets, down to 2 (16 lanes to each).  A power of
// two; tuned > 0: the next one from it, at least 2.
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
    // the coordinates' values of a constraint with several lanes are shared
    const size_t smem = local_terms_smem_bytes(per_warp)
        + (per_warp == kBarrierTPB ? 0 : (size_t)(kRed * kCoord) * (per_warp | 1) * sizeof(double));
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

static int body_frames(const double* x, int nb, double* frames, cudaStream_t st)
{
    RIGC_COUNT_LAUNCH();
    if (nb <= kWarpFrames) k_body_frames<true><<<grid_for((int64_t)nb * 32, 32), 32, 0, st>>>(x, nb, frames);
    else k_body_frames<false><<<grid_for(nb, 128), 128, 0, st>>>(x, nb, frames);
    RIGC_CUDA(cudaGetLastError());
    return RIGC_OK;
}

int launch_body_frames(Ctx& c, const double* x)
{
    RIGC_TRY(c.frames.reserve((size_t)c.s.nb * 96 * sizeof(double)));
    return body_frames(x, c.s.nb, c.frames.as<double>(), c.stream);
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
    RIGC_TRY(body_frames(x, nb, frames, stream));
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
// too.  (A constraint between vertices of one body, which a caller may set, has
// all four slots there: 4 c + 1 and 4 c + 2 add nothing to the gradient.)
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
            const uint32_t slot = slots[i], q = slot & 3;
            return q == 1 || q == 2 ? 0.0 : cgrad[(size_t)(slot >> 2) * 12 + 6 * (q == 3) + e];
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

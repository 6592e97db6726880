// Piecewise-linear trajectory CCD over EE and FV candidates.
//
// Replaces compute_earliest_toi_narrow_phase
// (src/opt/distance_barrier_constraint.cpp:151-265) with trajectory
// PIECEWISE_LINEAR: compute_piecewise_linear_edge_edge_time_of_impact and
// compute_piecewise_linear_face_vertex_time_of_impact
// (src/ccd/piecewise_linear/time_of_impact.cpp:326-651).  The time interval
// is cut into pieces over which each body's pose moves linearly
// (Pose::interpolate), the vertices move on straight lines between their
// positions at a piece's ends, and a linear CCD with a minimum separation
// (the interval bound of the rigid trajectory's deviation from the straight
// line, plus dmin) finds the first time the straight-line motions come that
// close.  Piece rules: an impact at the start of a piece whose features came
// below 0.2 of their initial distance (after t = 1e-6); a piece whose
// deviation is >= 0.5 of the features' distance at its start is halved
// (while fewer than 1000 halvings were made, or always at t = 0); an impact
// of the linear CCD at the piece's start halves the piece.
//
// The reference's linear CCD is Tight-Inclusion's inclusion-based root
// finder (Wang et al. 2021); the one here keeps its published method: the
// distance function F(t, u, v) of the straight-line motions is multilinear,
// so its range over a box is the hull of its values at the eight corners
// (evaluated in interval arithmetic); a box whose range misses [-ms, ms]^3
// holds no impact; one inside [-ms, ms]^3 or no wider than 1e-6 + ms in
// every coordinate is a root; others are halved along the dimension with the
// largest change of F between opposite corners, earlier half first; at most
// 10^6 boxes per piece (then the smallest unexplored t.lo, a conservative
// time).
//
// Two kernels.  k_pl_search (the default) takes the pieces of a candidate and
// the boxes of a piece as independent work items, a thread each: the piece
// logic in double precision, a box's decisions in single precision with an
// error bound and in double precision where that cannot tell.  k_pl_ccd takes
// one candidate per warp in double precision throughout: the search state is
// the same in every lane; a box's 8 corners x 3 coordinates are evaluated on
// 24 lanes (lane 8 j + k: coordinate j at corner k), the hull and the changes
// by shuffles; the piece's straight-line end points come from 4 lanes per end
// (one vertex each) and its deviation bound from 4 (one vertex each: its
// body's interval pose and rotation over the piece).  Every candidate
// searches t in [0, 1], the reference's first candidate's domain; the
// operations that decide are the oracle's, so the per-candidate times of
// impact are the same bits.
#include <algorithm>

#include "common.cuh"
#include "geometry_rn.cuh"
#include "interval.cuh"
#include "search_tree.cuh"

namespace rigc {

namespace {

constexpr int kPLThreads = 128;
constexpr double kLinearTol = 1e-6;
constexpr long long kLinearMaxBoxes = 1000000;
constexpr int kMaxSubdivisions = 1000;
constexpr int kMaxPieceDepth = 60;
constexpr double kTrajectoryFactor = 0.5;
constexpr double kDecreasingFactor = 0.2;
constexpr double kDecreasingMinTime = 1e-6;

// Every piece is a node of the dyadic bisection tree of [0, 1]
// ([k 2^-d, (k + 1) 2^-d]: the pieces are halvings of [0, 1] visited in order),
// and a body's interval frame over a piece and its rotation at a piece end
// depend on the body and the time only, not on the candidate.  So both are
// computed once per call for the pieces of depth < kPLTableDepth and their
// end points (k_pl_table) and shared by all the body's candidates; deeper
// pieces compute theirs on the spot.  The same operations either way.
constexpr int kPLTableDepth = 7;
constexpr int kPLNodes = (1 << kPLTableDepth) - 1;  // 127 pieces per body
constexpr int kPLPoints = (1 << (kPLTableDepth - 1)) + 1;  // 65 piece ends: k / 64
constexpr int kPLFrame = 24;                         // R (9 intervals) + p (3 intervals)

struct PLArgs {
    const double* rest;
    const int* edges;
    const int* faces;
    const int* vbody;
    const int* ebody;
    const int* fbody;
    const double* x0;
    const double* x1;
    const int2* ee;
    const int2* fv;
    int64_t nee, nfv;
    double dmin;
    double* per;                 // per-candidate time of impact (INFINITY: none)
    unsigned long long* gmin;    // earliest over all candidates (double bits)
    unsigned long long* next;    // next candidate
    unsigned long long* boxes;   // linear-CCD boxes over all candidates
    unsigned long long* pieces;  // pieces over all candidates
    int* status;                 // worst status
    const double* frames;        // per body: kPLNodes piece frames (kPLFrame doubles)
    const double* rots;          // per body: kPLPoints rotations at k / 64 (9 doubles)
    const int* list;             // k_pl_ccd: the candidates to take, or null (all)
    const unsigned long long* n_list;
};

// the interval pose of a body over a piece between the poses xa, xb (the
// piece's ends) and its interval rotation (time_of_impact.cpp:381-403)
__device__ void piece_frame(const double* xa, const double* xb, Itv R[9], Itv p[3])
{
    const Itv t { 0.0, 1.0 };
    Itv r[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        p[k] = iadd(imul_nonneg(isub(pt(xb[k]), pt(xa[k])), t), pt(xa[k]));
        r[k] = iadd(imul_nonneg(isub(pt(xb[3 + k]), pt(xa[3 + k])), t), pt(xa[3 + k]));
    }
    irotation(r, R);
}

// (x1 - x0) t + x0 per pose coordinate, round to nearest (Pose::interpolate)
__device__ __forceinline__ void pose_lerp(const double* x0, const double* x1, double t, double* x)
{
#pragma unroll
    for (int k = 0; k < 6; k++) x[k] = __dadd_rn(__dmul_rn(__dsub_rn(x1[k], x0[k]), t), x0[k]);
}

// thread per (body, slot): slots 0 .. kPLNodes-1 the piece frames of depth
// < kPLTableDepth, then the kPLPoints rotations at the piece ends
__global__ void k_pl_table(const double* __restrict__ x0, const double* __restrict__ x1, int nb,
                           double* __restrict__ frames, double* __restrict__ rots)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int per = kPLNodes + kPLPoints;
    if (i >= (int64_t)nb * per) return;
    const int b = (int)(i / per), slot = (int)(i % per);
    const double* xb0 = x0 + 6 * b;
    const double* xb1 = x1 + 6 * b;
    if (slot < kPLNodes) {
        const int d = 31 - __clz(slot + 1), k = slot + 1 - (1 << d);
        const double ta = ldexp((double)k, -d), tb = ldexp((double)(k + 1), -d);
        double xa[6], xc[6];
        pose_lerp(xb0, xb1, ta, xa);
        pose_lerp(xb0, xb1, tb, xc);
        Itv R[9], p[3];
        piece_frame(xa, xc, R, p);
        double* o = frames + ((size_t)b * kPLNodes + slot) * kPLFrame;
#pragma unroll
        for (int j = 0; j < 9; j++) {
            o[2 * j] = R[j].lo;
            o[2 * j + 1] = R[j].hi;
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            o[18 + 2 * j] = p[j].lo;
            o[19 + 2 * j] = p[j].hi;
        }
    } else {
        const int k = slot - kPLNodes;
        double x[6], R[9];
        pose_lerp(xb0, xb1, ldexp((double)k, -(kPLTableDepth - 1)), x);
        rot_rn(x + 3, R);
        double* o = rots + ((size_t)b * kPLPoints + k) * 9;
#pragma unroll
        for (int j = 0; j < 9; j++) o[j] = R[j];
    }
}

// the node of the piece [ti0, ti1]: pieces are aligned dyadic intervals
// (halvings of [0, 1] visited in order), so ti1 - ti0 = 2^-depth exactly and
// ti0 = k 2^-depth
__device__ __forceinline__ void piece_node(double ti0, double ti1, int& depth, long long& k)
{
    const double len = __dsub_rn(ti1, ti0);
    depth = 1023 - (int)((__double_as_longlong(len) >> 52) & 0x7ff);
    k = (long long)ldexp(ti0, depth);
}

// the frame of a body over the piece (node (1 << depth) + k) between the
// poses xa, xb: from the table for depth < kPLTableDepth
__device__ void body_piece_frame(const PLArgs& a, int body, int depth, long long k, const double* xa,
                                 const double* xb, Itv R[9], Itv p[3])
{
    if (depth < kPLTableDepth) {
        const double* e = a.frames + ((size_t)body * kPLNodes + (1 << depth) - 1 + k) * kPLFrame;
#pragma unroll
        for (int j = 0; j < 9; j++) R[j] = Itv { e[2 * j], e[2 * j + 1] };
#pragma unroll
        for (int j = 0; j < 3; j++) p[j] = Itv { e[18 + 2 * j], e[19 + 2 * j] };
        return;
    }
    piece_frame(xa, xb, R, p);
}

// the rotation of a body at the piece end t = e 2^-depth (pose x there): from
// the table when t is a multiple of 1/64
__device__ void body_point_rot(const PLArgs& a, int body, int depth, long long e, const double* x,
                               double R[9])
{
    if (depth < kPLTableDepth) {
        const double* o = a.rots + ((size_t)body * kPLPoints + (e << (kPLTableDepth - 1 - depth))) * 9;
#pragma unroll
        for (int j = 0; j < 9; j++) R[j] = o[j];
        return;
    }
    rot_rn(x + 3, R);
}

__device__ __forceinline__ double shfl(double v, int src)
{
    return __shfl_sync(0xffffffffu, v, src);
}

// (x1 - x0) t + x0, round to nearest
__device__ __forceinline__ double lerp_rn(double a, double b, double t)
{
    return RADD(RMUL(RSUB(b, a), t), a);
}

__device__ __forceinline__ double pt_sqdist_rn(const double* p, const double* t0, const double* t1,
                                               const double* t2)
{
    switch (pt_type_rn(p, t0, t1, t2)) {
    case PT_P_T0: return pp_sqdist_rn(p, t0);
    case PT_P_T1: return pp_sqdist_rn(p, t1);
    case PT_P_T2: return pp_sqdist_rn(p, t2);
    case PT_P_E0: return pl_sqdist_rn(p, t0, t1);
    case PT_P_E1: return pl_sqdist_rn(p, t1, t2);
    case PT_P_E2: return pl_sqdist_rn(p, t2, t0);
    default: return ptplane_sqdist_rn(p, t0, t1, t2);
    }
}

__device__ __forceinline__ double feature_distance(bool fv, const double P[4][3])
{
    return __dsqrt_rn(fv ? pt_sqdist_rn(P[0], P[1], P[2], P[3]) : ee_sqdist_rn(P[0], P[1], P[2], P[3]));
}

// Every lane gets the four points at the poses pa (body A) and pb (body B):
// lane m < 4 computes point m, the others take it by shuffles.
__device__ void gather_points(const PLArgs& a, const int vid[4], int na, int A, int B,
                              const double* pa, const double* pb, int depth, long long e, int lane,
                              double P[4][3])
{
    double w[3] = { 0, 0, 0 };
    if (lane < 4) {
        const double* x = lane < na ? pa : pb;
        double R[9], v[3];
        body_point_rot(a, lane < na ? A : B, depth, e, x, R);
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = a.rest[3 * (size_t)vid[lane] + c];
        world_vertex_rn(R, x, v, w);
    }
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int c = 0; c < 3; c++) P[m][c] = shfl(w[c], m);
}

// The largest deviation of each side's vertices from their straight lines
// over the piece between the poses at its ends (pa0 -> pa1, pb0 -> pb1):
// lane m < 4 bounds vertex m; returns the sum of the two sides' largest.
__device__ double piece_deviation(const PLArgs& a, const int vid[4], int na, int A, int B,
                                  const double* pa0, const double* pa1, const double* pb0,
                                  const double* pb1, int depth, long long k, const double P0[4][3],
                                  const double P1[4][3], int lane)
{
    double dev = 0;
    if (lane < 4) {
        const double* xa = lane < na ? pa0 : pb0;
        const double* xb = lane < na ? pa1 : pb1;
        const Itv t { 0.0, 1.0 };
        Itv p[3], R[9];
        body_piece_frame(a, lane < na ? A : B, depth, k, xa, xb, R, p);
        double v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = a.rest[3 * (size_t)vid[lane] + c];
        Itv w[3];
        iworld_vertex(R, p, v, w);
        Itv sq { 0.0, 0.0 };
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const Itv line = iadd(imul_nonneg(isub(pt(P1[lane][j]), pt(P0[lane][j])), t), pt(P0[lane][j]));
            const Itv e = isub(w[j], line);
            sq = j == 0 ? imul(e, e) : iadd(sq, imul(e, e));
        }
        dev = isqrt(sq).hi;
    }
    // largest of each side (lanes 0 .. na-1: A; na .. 3: B), then their sum
    double da = 0, db = 0;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const double d = shfl(dev, m);
        if (m < na) da = da < d ? d : da;
        else db = db < d ? d : db;
    }
    return RADD(da, db);
}

// The linear CCD of one piece by the warp: the first t in [0, 1] at which
// the straight-line motions P0 -> P1 come within ms (INFINITY: none).
__device__ double linear_toi(bool fv, const double P0[4][3], const double P1[4][3], double ms,
                             int lane, long long& boxes, int& status)
{
    // lanes < 24 in three roles per box, lane = 8 j + r for coordinate j:
    //  1. r = 4 it + m: point m's position at t = t_it (it 0: t0, 1: t1);
    //  2. r = 4 it + 2 iw + ab: the edge terms a(t_it, u_iw) (ab = 0) and
    //     b(t_it, v_iw) (ab = 1) of the distance function;
    //  3. r = k: F at corner k = it + 2 iu + 4 iv, b - a combined.
    // The same operations on the same operands as corner by corner.
    const int j = lane >> 3, k = lane & 7;
    const bool clane = lane < 24;
    const int it1 = (k >> 2) & 1, m1 = k & 3;         // role 1
    const int iw2 = (k >> 1) & 1, ab2 = k & 1;        // role 2 (it = it1)
    const int iu3 = (k >> 1) & 1, iv3 = (k >> 2) & 1, it3 = k & 1;  // role 3
    const double p0m = clane ? P0[m1][j] : 0.0, p1m = clane ? P1[m1][j] : 0.0;
    Node cn { { 0, 0, 0 }, { 0ull, 0ull, 0ull }, 0 };
    bool has_cn = true;
    u128 pend = 0, mt = 0, ma = 0;
    double earliest = INFINITY;
    long long n = 0;
    while (has_cn || pend != 0) {
        if (has_cn) {
            has_cn = false;
        } else {
            const int b = msb128(pend);
            pend &= ~bit128(b);
            cn = pending_node(cn, mt, ma, b);
        }
        const double t0 = dyadic(cn.ix[0], cn.lv[0]), t1 = dyadic(cn.ix[0] + 1, cn.lv[0]);
        const double u0 = dyadic(cn.ix[1], cn.lv[1]), u1 = dyadic(cn.ix[1] + 1, cn.lv[1]);
        const double v0 = dyadic(cn.ix[2], cn.lv[2]), v1 = dyadic(cn.ix[2] + 1, cn.lv[2]);
        if (t0 >= earliest) continue;
        if (fv && !(add_dn(u0, v0) <= 1.0)) continue;
        if (n >= kLinearMaxBoxes) {
            double m = t0;
            for (u128 r = pend; r != 0; r &= r - 1) {
                const Node g = pending_node(cn, mt, ma, lsb128(r));
                const double g0 = dyadic(g.ix[0], g.lv[0]);
                m = g0 < m ? g0 : m;
            }
            earliest = m < earliest ? m : earliest;
            status = status > 5 ? status : 5;
            break;
        }
        n++;
        // 1. the points at t0 and t1
        const Itv q = iadd(imul_nonneg(isub(pt(p1m), pt(p0m)), pt(it1 ? t1 : t0)), pt(p0m));
        // 2. the edge terms: EE a = (q1 - q0) u + q0, b = (q3 - q2) v + q2;
        //    FV a = (q2 - q1) u, b = (q3 - q1) v
        const int qb = 8 * j + 4 * it1;  // role-1 lanes of (j, t_it)
        const int sa = fv ? (ab2 ? 3 : 2) : (ab2 ? 3 : 1);
        const int sb = fv ? 1 : (ab2 ? 2 : 0);
        const Itv qa { __shfl_sync(0xffffffffu, q.lo, qb + sa), __shfl_sync(0xffffffffu, q.hi, qb + sa) };
        const Itv qs { __shfl_sync(0xffffffffu, q.lo, qb + sb), __shfl_sync(0xffffffffu, q.hi, qb + sb) };
        const Itv w = pt(ab2 ? (iw2 ? v1 : v0) : (iw2 ? u1 : u0));
        const Itv d = imul_nonneg(isub(qa, qs), w);
        const Itv term = fv ? d : iadd(d, qs);
        // 3. F at corner k
        const int tb0 = 8 * j + 4 * it3;  // role-2 and role-1 lanes of (j, t_it)
        const Itv ta { __shfl_sync(0xffffffffu, term.lo, tb0 + 2 * iu3), __shfl_sync(0xffffffffu, term.hi, tb0 + 2 * iu3) };
        const Itv tb { __shfl_sync(0xffffffffu, term.lo, tb0 + 2 * iv3 + 1),
                       __shfl_sync(0xffffffffu, term.hi, tb0 + 2 * iv3 + 1) };
        Itv y { 0.0, 0.0 };
        if (fv) {
            const Itv q0 { __shfl_sync(0xffffffffu, q.lo, tb0), __shfl_sync(0xffffffffu, q.hi, tb0) };
            const Itv q1 { __shfl_sync(0xffffffffu, q.lo, tb0 + 1), __shfl_sync(0xffffffffu, q.hi, tb0 + 1) };
            if (clane) y = isub(q0, iadd(iadd(ta, tb), q1));
        } else if (clane) {
            y = isub(ta, tb);
        }
        // the changes of F along t, u, v: |mid(corner with the bit) -
        // mid(corner without)|, largest over the lanes
        const double mid = RMUL(0.5, RADD(y.lo, y.hi));
        double ch[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double other = __shfl_xor_sync(0xffffffffu, mid, 1 << d);
            double c = (clane && !(k & (1 << d))) ? fabs(RSUB(other, mid)) : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double w = __shfl_xor_sync(0xffffffffu, c, o);
                c = c < w ? w : c;
            }
            ch[d] = c;
        }
        // hull over the corners of each coordinate (the 8 lanes of j)
        double lo = y.lo, hi = y.hi;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            const double l = __shfl_xor_sync(0xffffffffu, lo, o);
            const double h = __shfl_xor_sync(0xffffffffu, hi, o);
            lo = l < lo ? l : lo;
            hi = hi < h ? h : hi;
        }
        const bool meets_j = !clane || (lo <= ms && hi >= -ms);
        const bool inside_j = !clane || (lo >= -ms && hi <= ms);
        const bool small_j = !clane || sub_up(hi, lo) <= RADD(kLinearTol, ms);
        if (!__all_sync(0xffffffffu, meets_j)) continue;
        if (__all_sync(0xffffffffu, inside_j) || __all_sync(0xffffffffu, small_j)) {
            earliest = t0;
            continue;
        }
        int split = 0;
        if (ch[1] > ch[split]) split = 1;
        if (ch[2] > ch[split]) split = 2;
        if (cn.depth >= kMaxDepth || cn.lv[split] >= kMaxLevel) {
            earliest = t0;
            status = status > 4 ? status : 4;
            continue;
        }
        descend(cn, pend, mt, ma, split);
        has_cn = true;
    }
    boxes += n;
    return earliest;
}

// the piecewise-linear time of impact of one candidate (INFINITY: none)
__device__ double pl_toi(const PLArgs& a, bool fv, const int vid[4], int A, int B, int lane,
                         long long& boxes, long long& npieces, int& status)
{
    const int na = fv ? 1 : 2;
    const double* xa0 = a.x0 + 6 * A;
    const double* xa1 = a.x1 + 6 * A;
    const double* xb0 = a.x0 + 6 * B;
    const double* xb1 = a.x1 + 6 * B;
    double P0[4][3], P1[4][3];
    gather_points(a, vid, na, A, B, xa0, xb0, 0, 0, lane, P0);
    const double distance_t0 = feature_distance(fv, P0);
    if (distance_t0 <= a.dmin) return 0.0;
    double ts[kMaxPieceDepth + 1];
    int top = 0;
    ts[0] = 1.0;
    int subdivisions = 1;
    double ti0 = 0;
    double pa0[6], pb0[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        pa0[k] = xa0[k];
        pb0[k] = xb0[k];
    }
    double result = INFINITY;
    // the points and the distance at ti0 change only when a piece is passed
    // (a halving keeps ti0): P0 holds them for the current ti0
    double distance_ti0 = distance_t0;
    while (top >= 0) {
        const double ti1 = ts[top];
        double pa1[6], pb1[6];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            pa1[k] = lerp_rn(xa0[k], xa1[k], ti1);
            pb1[k] = lerp_rn(xb0[k], xb1[k], ti1);
        }
        if (distance_ti0 < RMUL(kDecreasingFactor, distance_t0) && ti0 >= kDecreasingMinTime) {
            result = ti0;
            break;
        }
        int depth;
        long long k;
        piece_node(ti0, ti1, depth, k);
        gather_points(a, vid, na, A, B, pa1, pb1, depth, k + 1, lane, P1);
        const double dev = piece_deviation(a, vid, na, A, B, pa0, pa1, pb0, pb1, depth, k, P0, P1, lane);
        const bool may_split = top < kMaxPieceDepth;
        if (dev >= RMUL(kTrajectoryFactor, distance_ti0) && (subdivisions < kMaxSubdivisions || ti0 == 0)) {
            if (!may_split) {
                result = ti0;
                status = status > 4 ? status : 4;
                break;
            }
            ts[++top] = RMUL(0.5, RADD(ti1, ti0));
            subdivisions++;
            continue;
        }
        const double t = linear_toi(fv, P0, P1, RADD(dev, a.dmin), lane, boxes, status);
        if (t < INFINITY) {
            const double tt = RADD(RMUL(RSUB(ti1, ti0), t), ti0);
            if (tt == 0) {
                if (!may_split) {
                    result = 0;
                    status = status > 4 ? status : 4;
                    break;
                }
                ts[++top] = RMUL(0.5, RADD(ti1, ti0));
                subdivisions++;
                continue;
            }
            result = tt;
            break;
        }
        top--;
        ti0 = ti1;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            pa0[k] = pa1[k];
            pb0[k] = pb1[k];
        }
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int c = 0; c < 3; c++) P0[m][c] = P1[m][c];
        distance_ti0 = feature_distance(fv, P0);
    }
    npieces += subdivisions;
    return result;
}

// ---------------------------------------------------------------------------
// Pieces and boxes as work items.  An FP64 warp instruction takes this GPU's
// FP64 unit 64 cycles whatever its active lanes, and a candidate is a chain of
// ten pieces on average and hundreds at worst, so one candidate per warp (or
// per lane: the last chains run alone) leaves the unit mostly idle:
//  * the pieces of a candidate are nodes of the bisection tree of [0, 1].  A
//    piece is halved by a rule on the piece alone, and the candidate's time of
//    impact is the first event in time order over the pieces, so all pieces
//    can be looked at in any order and the result is the smallest event time;
//    pieces that start at or after it are dropped;
//  * a piece's boxes (the linear CCD) are likewise a tree whose earliest root
//    does not depend on the visiting order;
//  * a block keeps stacks of pending pieces (those whose frames the table
//    holds, and deeper ones, which cost two interval rotations more) and of
//    pending boxes in shared memory and takes a batch of one kind at a time, a
//    thread per item, whatever the candidates;
//  * a box is decided in single precision (box32): the distance function is
//    multilinear, F = Z' - A' u - B' v with Z' = Z + Zt t, A' = A + At t,
//    B' = B + Bt t, and its corner values are its value at the lower corner,
//    in float pairs, plus differences that shrink with the box.  Every
//    decision (misses, root, dimension to halve) that the error bound leaves
//    open is taken by the double-precision evaluation of that box (box64):
//    one box in 10^4;
//  * what depends on the order after all (the caps on halvings and boxes, and
//    depths whose times are not exact here) sends the candidate to k_pl_ccd.
// Measured against one candidate per warp: a pile of 150 icospheres (93 k
// candidates, 0.92 M halvings, 6.6 M boxes) 128 -> 8.2 ms, 12 icospheres (6.5 k)
// 21.6 -> 1.6 ms, 27 resting cubes (1012) 60 -> 1.8 ms.  What is left is the
// FP64 of the pieces (~970 warp instructions per batch and warp).

__device__ __forceinline__ void lane_points(const PLArgs& a, const int vid[4], int na, int A, int B,
                                            const double* pa, const double* pb, int depth, long long e,
                                            double P[4][3])
{
    double RA[9], RB[9];
    body_point_rot(a, A, depth, e, pa, RA);
    body_point_rot(a, B, depth, e, pb, RB);
#pragma unroll
    for (int m = 0; m < 4; m++) {
        double v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = a.rest[3 * (size_t)vid[m] + c];
        world_vertex_rn(m < na ? RA : RB, m < na ? pa : pb, v, P[m]);
    }
}

// the largest deviation of one side's vertices m0 .. m1-1 over the piece
__device__ double lane_side_deviation(const PLArgs& a, const int vid[4], int m0, int m1, int body,
                                      const double* xa, const double* xb, int depth, long long k,
                                      const double P0[4][3], const double P1[4][3])
{
    const Itv t { 0.0, 1.0 };
    Itv p[3], R[9];
    body_piece_frame(a, body, depth, k, xa, xb, R, p);
    double dev = 0;
    for (int m = m0; m < m1; m++) {
        double v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = a.rest[3 * (size_t)vid[m] + c];
        Itv w[3];
        iworld_vertex(R, p, v, w);
        Itv sq { 0.0, 0.0 };
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const Itv line = iadd(imul_nonneg(isub(pt(P1[m][j]), pt(P0[m][j])), t), pt(P0[m][j]));
            const Itv e = isub(w[j], line);
            sq = j == 0 ? imul(e, e) : iadd(sq, imul(e, e));
        }
        const double d = isqrt(sq).hi;
        dev = dev < d ? d : dev;
    }
    return dev;
}

// what a box's evaluation decides: 0 no impact in it, 1 a root, 2 + d: halve
// it along dimension d; -1: not decided
__device__ int box64(bool fv, const double P0[4][3], const double P1[4][3],
                                              const Node& cn, double ms)
{
    const double t0 = dyadic(cn.ix[0], cn.lv[0]), t1 = dyadic(cn.ix[0] + 1, cn.lv[0]);
    const double u0 = dyadic(cn.ix[1], cn.lv[1]), u1 = dyadic(cn.ix[1] + 1, cn.lv[1]);
    const double v0 = dyadic(cn.ix[2], cn.lv[2]), v1 = dyadic(cn.ix[2] + 1, cn.lv[2]);
    // F at the 8 corners: the hull per coordinate and the corner midpoints.
    // The points' positions depend on t only and the edge (or face-edge)
    // terms on (t, u) or (t, v), so they are formed once per value and
    // combined per corner: the same operations on the same operands as
    // corner by corner.
    double mid[8][3], lo[3], hi[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        Itv q[2][4];
#pragma unroll
        for (int it = 0; it < 2; it++) {
            const Itv t = pt(it ? t1 : t0);
#pragma unroll
            for (int m = 0; m < 4; m++)
                q[it][m] = iadd(imul_nonneg(isub(pt(P1[m][j]), pt(P0[m][j])), t), pt(P0[m][j]));
        }
        // EE: a(t, u) = (q1 - q0) u + q0, b(t, v) = (q3 - q2) v + q2;
        // FV: a(t, u) = (q2 - q1) u, b(t, v) = (q3 - q1) v
        Itv ta[2][2], tb[2][2];
#pragma unroll
        for (int it = 0; it < 2; it++)
#pragma unroll
            for (int iw = 0; iw < 2; iw++) {
                const Itv u = pt(iw ? u1 : u0), v = pt(iw ? v1 : v0);
                const Itv* qt = q[it];
                if (fv) {
                    ta[it][iw] = imul_nonneg(isub(qt[2], qt[1]), u);
                    tb[it][iw] = imul_nonneg(isub(qt[3], qt[1]), v);
                } else {
                    ta[it][iw] = iadd(imul_nonneg(isub(qt[1], qt[0]), u), qt[0]);
                    tb[it][iw] = iadd(imul_nonneg(isub(qt[3], qt[2]), v), qt[2]);
                }
            }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int it = k & 1, iu = (k >> 1) & 1, iv = (k >> 2) & 1;
            const Itv y = fv ? isub(q[it][0], iadd(iadd(ta[it][iu], tb[it][iv]), q[it][1]))
                             : isub(ta[it][iu], tb[it][iv]);
            mid[k][j] = RMUL(0.5, RADD(y.lo, y.hi));
            if (k == 0) {
                lo[j] = y.lo;
                hi[j] = y.hi;
            } else {
                lo[j] = y.lo < lo[j] ? y.lo : lo[j];
                hi[j] = hi[j] < y.hi ? y.hi : hi[j];
            }
        }
    }
    double ch[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double c = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (k & (1 << d)) continue;
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const double x = fabs(RSUB(mid[k | (1 << d)][j], mid[k][j]));
                c = c < x ? x : c;
            }
        }
        ch[d] = c;
    }
    bool meets = true, inside = true, small = true;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        meets = meets && lo[j] <= ms && hi[j] >= -ms;
        inside = inside && lo[j] >= -ms && hi[j] <= ms;
        small = small && sub_up(hi[j], lo[j]) <= RADD(kLinearTol, ms);
    }
    if (!meets) return 0;
    if (inside || small) return 1;
    int split = 0;
    if (ch[1] > ch[split]) split = 1;
    if (ch[2] > ch[split]) split = 2;
    return 2 + split;
}

// a double as a float and a float remainder
struct Pair32 {
    float h, l;
};
__device__ __forceinline__ Pair32 pair32(double x)
{
    const float h = (float)x;
    return Pair32 { h, (float)(x - (double)h) };
}
// a + b exactly as s + e
__device__ __forceinline__ float two_sum32(float a, float b, float& e)
{
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
    return s;
}
// x + y t in pairs, t a float
__device__ __forceinline__ Pair32 pair_fma(Pair32 y, float t, Pair32 x)
{
    const float p = __fmul_rn(y.h, t);
    float e;
    const float s = two_sum32(x.h, p, e);
    return Pair32 { s, (e + __fmaf_rn(y.h, t, -p)) + __fmaf_rn(y.l, t, x.l) };
}

// A piece's straight-line motions for box32: y = Z' - A' u - B' v (the
// offsets as in ccd_filter.cuh), each with its change over the piece.
struct Lines32 {
    Pair32 Z[3], A[3], B[3], Zt[3], At[3], Bt[3];
    float ms, e0;
};

__device__ __forceinline__ void lines32(bool fv, const double P0[4][3], const double P1[4][3], double ms, Lines32& L)
{
    float m = 0.0f, W = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        double d[2][3];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const double* q[4] = { e ? P1[0] : P0[0], e ? P1[1] : P0[1], e ? P1[2] : P0[2], e ? P1[3] : P0[3] };
            d[e][0] = q[0][c] - (fv ? q[1][c] : q[2][c]);
            d[e][1] = (fv ? q[2][c] : q[0][c]) - q[1][c];
            d[e][2] = q[3][c] - (fv ? q[1][c] : q[2][c]);
#pragma unroll
            for (int k = 0; k < 4; k++) W = fmaxf(W, fabsf((float)q[k][c]));
        }
        L.Z[c] = pair32(d[0][0]);
        L.A[c] = pair32(d[0][1]);
        L.B[c] = pair32(d[0][2]);
        L.Zt[c] = pair32(d[1][0] - d[0][0]);
        L.At[c] = pair32(d[1][1] - d[0][1]);
        L.Bt[c] = pair32(d[1][2] - d[0][2]);
        m = fmaxf(m, fmaxf(fabsf(L.Z[c].h), fmaxf(fabsf(L.A[c].h), fabsf(L.B[c].h))));
        m = fmaxf(m, fmaxf(fabsf(L.Zt[c].h), fmaxf(fabsf(L.At[c].h), fabsf(L.Bt[c].h))));
    }
    L.ms = (float)ms;
    L.e0 = 1.1368683772161603e-13f * (2.0f * m + 2.0f * W);
}

// The decision of box64 in single precision, -1 when the error bound
// leaves it open.  Errors, u = 2^-24: the lower corner's value in pairs is
// within 2^-43 m of the exact one (m the largest offset; a pair holds 2^-48,
// its operations lose 2^-46 each), the differences to the other corners
// within 16 u S of theirs, S = wt (|Zt| + |At| + |Bt|) + wu |A'| + wv |B'|; the
// double-precision hull and changes lie within 2^-45 W of the exact ones (W
// the world coordinates' magnitude); ms rounds by u ms, the bounds by u of
// theirs.
__device__ __forceinline__ int box32(const Lines32& L, float t0, float wt, float u0, float wu, float v0, float wv)
{
    const float u16 = 9.5367431640625e-07f;  // 16 u
    bool meets = true, misses = false, inside = true, outside = false, small = true, large = false;
    float ch0 = 0.0f, ch1 = 0.0f, ch2 = 0.0f, Smax = 0.0f;
    const float tol = (float)kLinearTol + L.ms;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const Pair32 A = pair_fma(L.At[c], t0, L.A[c]), B = pair_fma(L.Bt[c], t0, L.B[c]);
        const Pair32 Z = pair_fma(L.Zt[c], t0, L.Z[c]);
        Pair32 b = pair_fma(Pair32 { -A.h, -A.l }, u0, Z);
        b = pair_fma(Pair32 { -B.h, -B.l }, v0, b);
        // differences from the lower corner
        const float dt = wt * __fmaf_rn(-L.At[c].h, u0, __fmaf_rn(-L.Bt[c].h, v0, L.Zt[c].h));
        const float du = -wu * A.h, dv = -wv * B.h;
        const float dtu = -(wt * wu) * L.At[c].h, dtv = -(wt * wv) * L.Bt[c].h;
        const float du1 = du + dtu, dv1 = dv + dtv;
        const float lo = fminf(fminf(0.0f, du) + fminf(0.0f, dv), dt + fminf(0.0f, du1) + fminf(0.0f, dv1));
        const float hi = fmaxf(fmaxf(0.0f, du) + fmaxf(0.0f, dv), dt + fmaxf(0.0f, du1) + fmaxf(0.0f, dv1));
        const float S = wt * (fabsf(L.Zt[c].h) + fabsf(L.At[c].h) + fabsf(L.Bt[c].h)) + wu * fabsf(A.h) + wv * fabsf(B.h);
        const float es = u16 * S, e = es + L.e0 + 1.1920928955078125e-07f * (L.ms + fabsf(b.h));
        const float yl = (b.h + lo) + b.l, yh = (b.h + hi) + b.l;
        misses = misses || yl - e > L.ms || yh + e < -L.ms;
        meets = meets && yl + e <= L.ms && yh - e >= -L.ms;
        inside = inside && yl - e >= -L.ms && yh + e <= L.ms;
        outside = outside || yl + e < -L.ms || yh - e > L.ms;
        const float ew = 2.0f * es + L.e0 + 2.384185791015625e-07f * tol;
        small = small && (hi - lo) + ew <= tol;
        large = large || (hi - lo) - ew > tol;
        ch0 = fmaxf(ch0, fmaxf(fmaxf(fabsf(dt), fabsf(dt + dtu)), fmaxf(fabsf(dt + dtv), fabsf(dt + dtu + dtv))));
        ch1 = fmaxf(ch1, fmaxf(fabsf(du), fabsf(du1)));
        ch2 = fmaxf(ch2, fmaxf(fabsf(dv), fabsf(dv1)));
        Smax = fmaxf(Smax, S);
    }
    if (misses) return 0;
    if (!meets) return -1;
    if (inside || small) return 1;
    if (!(outside && large)) return -1;
    const float ec = 2.0f * u16 * Smax + L.e0;
    if (fabsf(ch1 - ch0) <= ec) return -1;
    const float best = fmaxf(ch0, ch1);
    if (fabsf(ch2 - best) <= ec) return -1;
    return ch2 > best ? 4 : ch1 > ch0 ? 3 : 2;
}

// the candidate's vertices (EE: a0 a1 b0 b1; FV: v f0 f1 f2) and bodies
__device__ __forceinline__ bool pl_candidate(const PLArgs& a, int64_t w, int vid[4], int& A, int& B)
{
    if (w < a.nee) {
        const int ea = a.ee[w].x, eb = a.ee[w].y;
        vid[0] = a.edges[2 * ea];
        vid[1] = a.edges[2 * ea + 1];
        vid[2] = a.edges[2 * eb];
        vid[3] = a.edges[2 * eb + 1];
        A = a.ebody[ea];
        B = a.ebody[eb];
        return false;
    }
    const int f = a.fv[w - a.nee].x, v = a.fv[w - a.nee].y;
    vid[0] = v;
    vid[1] = a.faces[3 * f];
    vid[2] = a.faces[3 * f + 1];
    vid[3] = a.faces[3 * f + 2];
    A = a.vbody[v];
    B = a.fbody[f];
    return true;
}

constexpr int kSearchThreads = 256;
constexpr int kPieceStack = 1280;   // pending pieces per block, of either kind
constexpr int kBoxStack = 3072;
constexpr int kJobs = 1024;         // pieces whose boxes are being searched, per block
constexpr int kExactDepth = 28;     // piece depth + 24 box levels stay exact doubles
constexpr int kBoxLevels = 24;
constexpr int kHard = 1 << 30;      // flag in nboxes: the candidate goes to k_pl_ccd
constexpr int kHardBoxes = 1 << 16; // boxes per candidate after which it does

struct PieceNode {
    int cand, depth;
    long long k;                    // [k, k + 1] 2^-depth
};
struct BoxNode {
    int job;
    unsigned x[3];                  // index (24 bits), level of t, u, v
};
struct alignas(16) Job {
    Lines32 L;
    int cand, depth, fv;
    long long k;
};

struct SearchArgs {
    double* d0;                     // per candidate: distance at t = 0
    unsigned long long* result;     // time of impact (double bits)
    int* halvings;
    int* nboxes;                    // boxes, kHard
    Job* jobs;                      // gridDim x kJobs
    int* hard;                      // candidates for k_pl_ccd
    unsigned long long* n_hard;
    int per_batch;                  // candidates a block starts on at a time
};

__device__ void mark_hard(const SearchArgs& s, int c)
{
    if (!(atomicOr(&s.nboxes[c], kHard) & kHard)) s.hard[atomicAdd(s.n_hard, 1ull)] = c;
}

// the points at both ends of a piece and the deviation bound over it
// (piece_deviation's operations)
__device__ __noinline__ double piece_ends(const PLArgs& a, bool fv, const int vid[4], int A, int B, int depth,
                                          long long k, double P0[4][3], double P1[4][3])
{
    const int na = fv ? 1 : 2;
    const double *xa0 = a.x0 + 6 * A, *xa1 = a.x1 + 6 * A, *xb0 = a.x0 + 6 * B, *xb1 = a.x1 + 6 * B;
    double pa[2][6], pb[2][6];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const double t = dyadic((unsigned long long)(k + e), depth);
#pragma unroll
        for (int q = 0; q < 6; q++) {
            pa[e][q] = lerp_rn(xa0[q], xa1[q], t);
            pb[e][q] = lerp_rn(xb0[q], xb1[q], t);
        }
    }
    lane_points(a, vid, na, A, B, pa[0], pb[0], depth, k, P0);
    lane_points(a, vid, na, A, B, pa[1], pb[1], depth, k + 1, P1);
    return RADD(lane_side_deviation(a, vid, 0, na, A, pa[0], pa[1], depth, k, P0, P1),
                lane_side_deviation(a, vid, na, 4, B, pb[0], pb[1], depth, k, P0, P1));
}

enum PieceStep { kPieceDone, kPieceHalve, kPieceBoxes };

// One piece: an event (recorded in result), a halving, or its boxes next
// (job filled).
__device__ __noinline__ PieceStep piece_step(const PLArgs& a, const SearchArgs& s, const PieceNode& p, Job& job)
{
    int vid[4], A, B;
    const bool fv = pl_candidate(a, p.cand, vid, A, B);
    double P0[4][3], P1[4][3];
    const double dev = piece_ends(a, fv, vid, A, B, p.depth, p.k, P0, P1);
    const double dist = feature_distance(fv, P0);
    double d0 = dist;
    if (p.depth == 0) {
        s.d0[p.cand] = dist;
        if (dist <= a.dmin) {
            atomicMin(&s.result[p.cand], 0ull);
            return kPieceDone;
        }
    } else {
        d0 = s.d0[p.cand];
    }
    const double ti0 = dyadic((unsigned long long)p.k, p.depth);
    if (dist < RMUL(kDecreasingFactor, d0) && ti0 >= kDecreasingMinTime) {
        atomicMin(&s.result[p.cand], (unsigned long long)__double_as_longlong(ti0));
        return kPieceDone;
    }
    if (dev >= RMUL(kTrajectoryFactor, dist)) return kPieceHalve;
    lines32(fv, P0, P1, RADD(dev, a.dmin), job.L);
    job.cand = p.cand;
    job.depth = p.depth;
    job.fv = fv ? 1 : 0;
    job.k = p.k;
    return kPieceBoxes;
}

// a box in double precision, from its piece
__device__ __noinline__ int box_exact(const PLArgs& a, const Job& job, const BoxNode& x)
{
    int vid[4], A, B;
    const bool fv = pl_candidate(a, job.cand, vid, A, B);
    double P0[4][3], P1[4][3];
    const double dev = piece_ends(a, fv, vid, A, B, job.depth, job.k, P0, P1);
    Node n;
    for (int d = 0; d < 3; d++) {
        n.lv[d] = (int)(x.x[d] >> 24);
        n.ix[d] = x.x[d] & 0xffffffu;
    }
    n.depth = 0;
    return box64(fv, P0, P1, n, RADD(dev, a.dmin));
}

// The block's sum of each thread's value and the threads' exclusive prefix
// (buf: one int per warp; two barriers apart from its last use)
__device__ __forceinline__ int block_rank(bool mine, int* buf, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) buf[warp] = __popc(m);
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int k = 0; k < kSearchThreads / 32; k++) {
        const int q = buf[k];
        if (k < warp) before += q;
        total += q;
    }
    return before + __popc(m & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(kSearchThreads, 2) k_pl_search(PLArgs a, SearchArgs s)
{
    extern __shared__ char smem_[];
    PieceNode* pieces[2];           // table depths, deeper
    pieces[0] = reinterpret_cast<PieceNode*>(smem_);
    pieces[1] = pieces[0] + kPieceStack;
    BoxNode* boxes = reinterpret_cast<BoxNode*>(pieces[1] + kPieceStack);
    int* pending = reinterpret_cast<int*>(boxes + kBoxStack);        // boxes left, per job
    unsigned* root = reinterpret_cast<unsigned*>(pending + kJobs);   // earliest root, 2^-24 units (~0: none)
    int* free_jobs = reinterpret_cast<int*>(root + kJobs);
    __shared__ int buf[4][kSearchThreads / 32];
    __shared__ int n_free_;
    __shared__ unsigned long long batch;
    const int tid = threadIdx.x;
    Job* jobs = s.jobs + (size_t)blockIdx.x * kJobs;
    const int64_t n = a.nee + a.nfv;
    const unsigned long long batches = (unsigned long long)((n + s.per_batch - 1) / s.per_batch);
    for (int i = tid; i < kJobs; i += kSearchThreads) free_jobs[i] = i;
    if (tid == 0) n_free_ = kJobs;
    __syncthreads();
    int np[2] = { 0, 0 }, nb = 0;   // stack heights (the same in every thread)
    bool more = true;
    long long tot_boxes = 0, tot_pieces = 0;
    while (true) {
        const int n_free = n_free_;
        // what to take a batch of: full batches first, then new candidates,
        // then what is left (boxes first: they free their jobs)
        const bool room = n_free >= kSearchThreads;
        int kind;                   // 0 / 1 pieces, 2 boxes, 3 new candidates
        if (nb >= kSearchThreads || nb > kBoxStack - 4 * kSearchThreads) kind = 2;
        else if (np[1] >= kSearchThreads && room) kind = 1;
        else if (np[0] >= kSearchThreads && room) kind = 0;
        else if (more && room) kind = 3;  // both below a batch: room for its halves
        else if (nb > 0) kind = 2;
        else if (np[0] > 0) kind = 0;
        else if (np[1] > 0) kind = 1;
        else if (more) kind = 3;
        else break;
        __syncthreads();            // n_free_ is read
        if (kind == 2) {
            // fewer at a time when the stack fills: depth first
            const int take = min(min(nb, kSearchThreads), (kBoxStack - nb) / 2 + 1);
            const bool mine = tid < take;
            BoxNode x { 0, { 0, 0, 0 } };
            if (mine) x = boxes[nb - 1 - tid];
            nb -= take;
            int what = 0;           // box64's decisions
            int again = -1;         // the piece to halve after all (its job)
            const Job& job = jobs[x.job];
            if (mine) {
                const int lt = (int)(x.x[0] >> 24), lu = (int)(x.x[1] >> 24), lv = (int)(x.x[2] >> 24);
                const unsigned it = x.x[0] & 0xffffffu, iu = x.x[1] & 0xffffffu, iv = x.x[2] & 0xffffffu;
                const unsigned t0 = it << (kBoxLevels - lt);
                // boxes from the job's earliest root on are skipped, as are
                // those of face-vertex pairs with u + v above 1 (add_dn of the
                // lower ends, an exact sum) and those of candidates given up
                const bool keep = t0 < *(volatile unsigned*)&root[x.job]
                    && !(job.fv && (iu << (kBoxLevels - lu)) + (iv << (kBoxLevels - lv)) > (1u << kBoxLevels));
                if (keep) {
                    const int seen = atomicAdd(&s.nboxes[job.cand], 1);
                    if (!(seen & kHard)) {
                        tot_boxes++;
                        const float wt = __int_as_float((127 - lt) << 23), wu = __int_as_float((127 - lu) << 23);
                        const float wv = __int_as_float((127 - lv) << 23);
                        what = box32(job.L, (float)it * wt, wt, (float)iu * wu, wu, (float)iv * wv, wv);
                        if (what < 0) what = box_exact(a, job, x);
                        const int l = what == 2 ? lt : what == 3 ? lu : lv;
                        if (seen >= kHardBoxes || (what >= 2 && l >= kBoxLevels - 1)) {
                            mark_hard(s, job.cand);
                            what = 0;
                        }
                        if (what == 1) atomicMin(&root[x.job], t0);
                    }
                }
            }
            const bool split = what >= 2;
            int ns;
            const int rank = block_rank(split, buf[0], ns);  // its barrier: the boxes are read
            bool lost = false;
            if (nb + 2 * ns <= kBoxStack) {
                if (split) {
                    const int d = what - 2;
                    BoxNode lo = x;
#pragma unroll
                    for (int q = 0; q < 3; q++)
                        if (q == d) lo.x[q] = (x.x[q] & 0xff000000u) + (1u << 24) + 2u * (x.x[q] & 0xffffffu);
                    BoxNode hi = lo;
#pragma unroll
                    for (int q = 0; q < 3; q++)
                        if (q == d) hi.x[q] |= 1u;
                    boxes[nb + ns - 1 - rank] = hi;
                    boxes[nb + 2 * ns - 1 - rank] = lo;
                }
                nb += 2 * ns;
            } else {
                lost = split;
            }
            if (lost) mark_hard(s, job.cand);
            if (mine) {
                const int left = atomicAdd(&pending[x.job], split && !lost ? 1 : -1) + (split && !lost ? 1 : -1);
                if (left == 0) {
                    // the piece's boxes are searched
                    const unsigned t = *(volatile unsigned*)&root[x.job];
                    if (t != ~0u) {
                        if (t == 0 && job.k == 0) again = x.job;
                        else
                            atomicMin(&s.result[job.cand],
                                      (unsigned long long)dbits(dyadic(((unsigned long long)job.k << kBoxLevels) + t,
                                                                       job.depth + kBoxLevels)));
                    }
                    if (again < 0) free_jobs[atomicAdd(&n_free_, 1)] = x.job;
                }
            }
            // an impact at t = 0 halves the piece
            PieceNode c { 0, 0, 0 };
            bool halve = again >= 0;
            if (halve) {
                c = PieceNode { jobs[again].cand, jobs[again].depth + 1, 0 };
                free_jobs[atomicAdd(&n_free_, 1)] = again;
                if (c.depth > kExactDepth || atomicAdd(&s.halvings[c.cand], 1) >= kMaxSubdivisions - 2) {
                    mark_hard(s, c.cand);
                    halve = false;
                }
            }
            if (__syncthreads_or(halve)) {
#pragma unroll
                for (int deep = 0; deep < 2; deep++) {
                    int nh;
                    const bool put = halve && (c.depth >= kPLTableDepth) == (deep == 1);
                    const int r = block_rank(put, buf[1 + deep], nh);
                    if (np[deep] + 2 * nh <= kPieceStack) {
                        if (put) {
                            pieces[deep][np[deep] + 2 * r] = PieceNode { c.cand, c.depth, 1 };
                            pieces[deep][np[deep] + 2 * r + 1] = c;
                        }
                        np[deep] += 2 * nh;
                    } else if (put) {
                        mark_hard(s, c.cand);
                    }
                }
            }
        } else {
            PieceNode p { 0, 0, 0 };
            bool mine = false;
            if (kind == 3) {
                if (tid == 0) batch = atomicAdd(a.next, 1ull);
                __syncthreads();
                if (batch >= batches) more = false;
                // a batch from distant places of the list, so that the
                // candidates of one contact spread over the blocks
                const int64_t c = (int64_t)batch + (int64_t)tid * (int64_t)batches;
                mine = more && tid < s.per_batch && c < n;
                p.cand = (int)c;
            } else {
                // fewer at a time when a stack they may go to fills
                const int space = min(kPieceStack - np[1], kPieceStack - np[kind]);
                const int take = min(min(np[kind], kSearchThreads), min(n_free, space / 2 + 1));
                mine = tid < take;
                if (mine) p = pieces[kind][np[kind] - 1 - tid];
                np[kind] -= take;
            }
            // jobs for the batch, one per thread, the unused given back
            const int ticket = n_free - 1 - tid;
            const int j = ticket >= 0 ? free_jobs[ticket] : -1;
            PieceStep step = kPieceDone;
            if (mine && !(*(volatile int*)&s.nboxes[p.cand] & kHard)
                && (unsigned long long)dbits(dyadic((unsigned long long)p.k, p.depth))
                    < *(volatile unsigned long long*)&s.result[p.cand]) {
                tot_pieces++;
                step = j < 0 ? kPieceHalve : piece_step(a, s, p, jobs[j]);
                if (step == kPieceHalve
                    && (j < 0 || p.depth >= kExactDepth
                        || atomicAdd(&s.halvings[p.cand], 1) >= kMaxSubdivisions - 2)) {
                    mark_hard(s, p.cand);
                    step = kPieceDone;
                }
            }
            int nj, nh;
            const bool boxed = step == kPieceBoxes;
            const int r = block_rank(boxed, buf[0], nj);  // its barrier: the stacks are read
            if (nb + nj <= kBoxStack) {
                if (boxed) {
                    boxes[nb + nj - 1 - r] = BoxNode { j, { 0, 0, 0 } };
                    pending[j] = 1;
                    root[j] = ~0u;
                }
                nb += nj;
            } else if (boxed) {
                mark_hard(s, p.cand);  // cannot happen: a batch of boxes is taken first
            }
            // the jobs kept move off the free list: the last n_free - take
            // slots stay, the batch's unused ones close up
            const int used = min(kSearchThreads, n_free);
            const bool unused = j >= 0 && !boxed;
            int nu;
            const int ru = block_rank(unused, buf[1], nu);
            if (unused) free_jobs[n_free - used + ru] = j;
            if (tid == 0) n_free_ = n_free - used + nu;
#pragma unroll
            for (int deep = 0; deep < 2; deep++) {
                const bool put = step == kPieceHalve && (p.depth + 1 >= kPLTableDepth) == (deep == 1);
                const int q = block_rank(put, buf[2 + deep], nh);
                if (np[deep] + 2 * nh <= kPieceStack) {
                    if (put) {
                        pieces[deep][np[deep] + 2 * (nh - 1 - q)] = PieceNode { p.cand, p.depth + 1, 2 * p.k + 1 };
                        pieces[deep][np[deep] + 2 * (nh - 1 - q) + 1] = PieceNode { p.cand, p.depth + 1, 2 * p.k };
                    }
                    np[deep] += 2 * nh;
                } else if (put) {
                    mark_hard(s, p.cand);
                }
            }
        }
        __syncthreads();            // the stacks are written
    }
    atomicAdd(a.boxes, (unsigned long long)tot_boxes);
    atomicAdd(a.pieces, (unsigned long long)tot_pieces);
}

size_t search_smem_bytes()
{
    return 2 * kPieceStack * sizeof(PieceNode) + kBoxStack * sizeof(BoxNode) + kJobs * 3 * sizeof(int);
}

__global__ void k_pl_init(SearchArgs s, int64_t n)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    s.result[i] = 0x7ff0000000000000ull;
    s.halvings[i] = 0;
    s.nboxes[i] = 0;
}

// the earliest time over the candidates k_pl_search finished
__global__ void k_pl_min(SearchArgs s, int64_t n, unsigned long long* gmin)
{
    unsigned long long m = 0x7ff0000000000000ull;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (!(s.nboxes[i] & kHard)) m = min(m, s.result[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m != 0x7ff0000000000000ull) atomicMin(gmin, m);
}

__global__ void __launch_bounds__(kPLThreads) k_pl_ccd(PLArgs a)
{
    const int lane = threadIdx.x & 31;
    const int64_t n = a.list ? (int64_t)*a.n_list : a.nee + a.nfv;
    long long boxes = 0, npieces = 0;
    int status = RIGC_OK;
    double local_min = INFINITY;
    while (true) {
        long long w = 0;
        if (lane == 0) w = (long long)atomicAdd(a.next, 1ull);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= n) break;
        if (a.list) w = a.list[w];
        int vid[4], A, B;
        const bool fv = pl_candidate(a, w, vid, A, B);
        const double toi = pl_toi(a, fv, vid, A, B, lane, boxes, npieces, status);
        if (lane == 0 && a.per) a.per[w] = toi;
        local_min = toi < local_min ? toi : local_min;
    }
    if (lane == 0) {
        if (local_min < INFINITY) atomicMin(a.gmin, (unsigned long long)__double_as_longlong(local_min));
        atomicAdd(a.boxes, (unsigned long long)boxes);
        atomicAdd(a.pieces, (unsigned long long)npieces);
        if (status != RIGC_OK) atomicMax(a.status, status);
    }
}

} // namespace

// counters in the context's device scalars (byte offset 512): [0] earliest
// time of impact (bits), [1] boxes, [2] pieces, [3] status, [4] next, [5]
// candidates k_pl_search left to k_pl_ccd, [6] the next of them
int run_pl_ccd(Ctx& c, const double* x0, const double* x1, double dmin, double* toi_host, double* per)
{
    cudaStream_t st = c.stream;
    const int64_t n = c.cand.num_ee + c.cand.num_fv;
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(c.d_scalars.as<char>() + 512);
    const unsigned long long init[7] = { 0x7ff0000000000000ull };
    RIGC_CUDA(cudaMemcpyAsync(cnt, init, sizeof(init), cudaMemcpyHostToDevice, st));
    if (n > 0) {
        PLArgs a;
        a.rest = c.s.rest;
        a.edges = c.s.edges;
        a.faces = c.s.faces;
        a.vbody = c.s.vbody;
        a.ebody = c.s.ebody;
        a.fbody = c.s.fbody;
        a.x0 = x0;
        a.x1 = x1;
        a.ee = c.cand.ee.as<int2>();
        a.fv = c.cand.fv.as<int2>();
        a.nee = c.cand.num_ee;
        a.nfv = c.cand.num_fv;
        a.dmin = dmin;
        a.per = per;
        a.gmin = cnt;
        a.boxes = cnt + 1;
        a.pieces = cnt + 2;
        a.status = reinterpret_cast<int*>(cnt + 3);
        a.next = cnt + 4;
        const size_t frame_doubles = (size_t)c.s.nb * kPLNodes * kPLFrame;
        RIGC_TRY(c.pl_table.reserve((frame_doubles + (size_t)c.s.nb * kPLPoints * 9) * sizeof(double)));
        a.frames = c.pl_table.as<double>();
        a.rots = c.pl_table.as<double>() + frame_doubles;
        RIGC_COUNT_LAUNCH();
        k_pl_table<<<grid_for((int64_t)c.s.nb * (kPLNodes + kPLPoints), 128), 128, 0, st>>>(
            x0, x1, c.s.nb, const_cast<double*>(a.frames), const_cast<double*>(a.rots));
        int dev = 0, sms = kNumSMs;
        RIGC_CUDA(cudaGetDevice(&dev));
        RIGC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        // pieces and boxes as work items unless tuned to one candidate per
        // warp (slower on every workload measured: k_pl_search's header)
        bool search = c.tune.pl_per_lane != 0 && n < (int64_t(1) << 31);
        a.list = nullptr;
        a.n_list = nullptr;
        int blocks = 0;
        RIGC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_pl_ccd, kPLThreads, 0));
        const unsigned full = (unsigned)(sms * std::max(1, blocks));
        unsigned grid = (unsigned)std::min<int64_t>((n + 3) / 4, full);
        // few candidates spread over all blocks, four or more to each
        const int per_batch = (int)std::max<int64_t>(4, std::min<int64_t>(kSearchThreads, (n + 2 * sms - 1) / (2 * sms)));
        const unsigned sblocks = (unsigned)std::min<int64_t>((n + per_batch - 1) / per_batch, 2 * sms);
        const size_t job_bytes = (size_t)sblocks * kJobs * sizeof(Job);
        // no memory for their state: one candidate per warp
        if (search) search = c.pl_work.reserve(job_bytes + (size_t)n * (2 * sizeof(double) + 3 * sizeof(int))) == RIGC_OK;
        if (search) {
            SearchArgs s;
            s.jobs = c.pl_work.as<Job>();
            s.d0 = reinterpret_cast<double*>(c.pl_work.as<char>() + job_bytes);
            s.result = per ? reinterpret_cast<unsigned long long*>(per) : reinterpret_cast<unsigned long long*>(s.d0 + n);
            s.halvings = reinterpret_cast<int*>(s.d0 + 2 * n);
            s.nboxes = s.halvings + n;
            s.hard = s.nboxes + n;
            s.n_hard = cnt + 5;
            s.per_batch = per_batch;
            // (the device's own attribute: set on each call, whichever device that is for)
            RIGC_CUDA(cudaFuncSetAttribute(k_pl_search, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)search_smem_bytes()));
            RIGC_COUNT_LAUNCH();
            k_pl_init<<<grid_for(n, 256), 256, 0, st>>>(s, n);
            RIGC_COUNT_LAUNCH();
            k_pl_search<<<sblocks, kSearchThreads, search_smem_bytes(), st>>>(a, s);
            RIGC_COUNT_LAUNCH();
            k_pl_min<<<std::min(grid_for(n, 256), (unsigned)(4 * sms)), 256, 0, st>>>(s, n, a.gmin);
            // the candidates it left
            a.next = cnt + 6;
            a.list = s.hard;
            a.n_list = s.n_hard;
            grid = full;
        }
        RIGC_COUNT_LAUNCH();
        k_pl_ccd<<<grid, kPLThreads, 0, st>>>(a);
        RIGC_CUDA(cudaGetLastError());
    }
    unsigned long long out[4];
    RIGC_CUDA(cudaMemcpyAsync(out, cnt, sizeof(out), cudaMemcpyDeviceToHost, st));
    RIGC_CUDA(cudaStreamSynchronize(st));
    double g;
    std::memcpy(&g, &out[0], sizeof(g));
    *toi_host = g;
    c.stats.ccd_boxes = (int64_t)out[1];
    c.stats.ccd_candidates = n;
    c.stats.last_status = (int)(out[3] & 0xffffffffu);
    return c.stats.last_status;
}

} // namespace rigc

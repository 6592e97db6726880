// Single-precision search of the pruned interval CCD (included by ccd.cu).
//
// k_ccd_filter walks each candidate's subdivision tree and decides each box
// with single-precision interval bounds and a bound E on how far they can be
// from the double-precision ones of f_zero:
//  * a bound beyond E excludes zero in double too: the box is dropped, as the
//    double-precision search drops it;
//  * a box within tolerance whose bounds include zero by more than E is a
//    root in double too, and its start lowers the running minimum;
//  * a box within tolerance in between, or starting at t = 0, or a level
//    beyond kFilterLevel, is written out as a search piece, and the
//    double-precision kernels decide it;
//  * any other box is split by the search's own rule.
// What single precision cannot decide is bounded: where the bodies do not move
// along an axis and the offset there is 0 (a box landing on or sliding along
// another, parallel edges), that axis's bounds are within E whatever the box's
// size, no box is ever a root, and at gaps below E none is dropped either.  So a
// candidate with kUndecidedLimit undecided boxes goes to the double-precision
// search from its seeds, and its other boxes and pieces are dropped; a launch
// whose pieces run over their buffer ends (the call is redone without it).
// Parallel 1 m edges, 0.1 m along one another at a gap of 1e-7 m: above 2^28
// boxes without the limit, 9000 with it (a block's boxes in flight when the first
// reach the tolerance).
// A box kept here that double precision would have dropped only costs its
// subtree: the interval operations are inclusion isotonic, so the boxes
// inside it are not roots.
//
// What bounds it: an FP64 warp instruction takes 64 cycles of its
// sub-partition on this GPU, a single-precision one 1, so the ~260 FP64
// operations of a box (or the ~900 warp instructions that spread them over a
// warp) become ~400 single-precision ones of a thread, a box per thread.  What is
// left is the latency of a block's turns: 16 to 23 % of the issue slots are used, the
// warps wait at the two barriers of a turn and for records and frames.
// Measured (device time of the search, double-precision kernels alone and
// with this one in front): a pile of 1000 icospheres, 709 k candidates, 20.4
// -> 0.84 ms (5.4 M boxes); a 200-link chain in contact, 41 k candidates, 6 ->
// 0.25 ms; 48 batched hull piles, 21 k candidates, 4.4 -> 0.86 ms; 27 resting
// cubes, 1012 candidates, 1.2 -> 0.2 ms.
//
// Layout: a block keeps its pending boxes in a stack of 16-byte nodes in
// shared memory, pops one per thread at a time (whatever their candidates: no
// thread waits for another's search) and pushes both halves of each kept
// box, lower halves on top.  Boxes that start at or after the first time
// window 2^-k wait in the block's lists in global memory, one per power of
// two of their start, and are searched list by list, so that all candidates'
// early boxes come first and the running minimum skips most of the others.
// A box reads its candidate's 128-byte record (FilterRec) and the two bodies'
// frames of its time node: 96 bytes each from a table of the nodes of depth
// < 7, computed by the thread from 96 bytes per body below that (deep_frame).
//
// With X_v(t) = C_v + d_v(t), C_v the vertex at the bodies' start poses and
// d_v = dp + dR v its displacement, the distance function of both kinds is
//   y = Z - A alpha - B beta + d_0 - d_k - F alpha - G beta,
// EE: Z = C0 - C2, A = C0 - C1, B = C3 - C2, k = 2, F = d0 - d1, G = d3 - d2;
// FV: Z = C0 - C1, A = C2 - C1, B = C3 - C1, k = 1, F = d2 - d1, G = d3 - d1.
// Z, A, B come from double once per candidate, as a float and a bfloat16
// remainder; Z - A alpha0 - B beta0 is evaluated in float pairs at the box's
// lower corner and the rest is small: displacements, and A and B times the
// box's widths.  So single precision rounds displacements and box sizes, not
// positions.
//
// Error bound, u = 2^-24.  Let D bound every displacement's |dp| + sum |dR||v|
// over t in [0, 1] (the root's frame contains all others).  Inputs and the
// six operations of a displacement give 8 u D; F, G 18 u D; their products
// with a coordinate of [0, 1] 20 u D, with A times a width added 4 u |A| w
// more; the sum of two displacements and two such terms 70 u D + 8 u (|A| w_a
// + |B| w_b).  Minima and maxima add nothing, the last sum rounds relative to
// its result.  The pairs hold Z, A, B to 2^-33, the corner to 2^-30 of the
// largest, m.  The double-precision bounds lie within 2^-45 W of the exact
// ones, W the world coordinates' magnitude.  deep_frame's entries are within
// 20 u T of the exact bounds (T: see there), which six times |v|_1 20 u T
// covers in the distance.  So with
//   E = 96 u D + 120 u max |v|_1 T + 2^-30 m + 2^-43 W
// the bounds are within E + 8 u (|A| w_a + |B| w_b).
#pragma once

#include <cuda_bf16.h>

namespace rigc {

constexpr int kFilterLevel = 24;     // levels whose bounds single precision holds exactly
constexpr int kFilterThreads = 256;
constexpr int kFilterBlocks = 3;     // resident per SM
constexpr int kFilterStack = 2048;   // pending boxes per block
constexpr int kFilterLists = 8;      // lists of later boxes per block
constexpr int kFrame32 = 24;         // m (9), radius (9), dp middle (3), radius (3)
constexpr int kRef64 = 12;           // start frame: R (9), p (3)
constexpr int kBody32 = 24;          // deep_frame's body: theta, dtheta, dp (3 each), S, C (6 each), T
constexpr int kTaylor = 6;           // terms of S and C about the start pose
constexpr int kSeries = 20;
constexpr float kMaxTheta = 4.4f;    // S decreases up to 4.493
// a candidate's state: undecided boxes from bit 32 on (kUndecidedLeaf for one
// within tolerance, 1 for a subtree: at the limit of the levels, or without room
// on the stack), bit 63 set once it is handed on.  The limit: over piles, cubes
// and chains (tilted contacts) a candidate has at most 20 within tolerance, nearly
// all none.
constexpr unsigned kUndecidedLeaf = 16, kUndecidedLimit = 64 * kUndecidedLeaf;
constexpr unsigned long long kHandedOn = 1ull << 63;

struct alignas(16) FilterRec {
    float v[4][3];                   // rest vertices
    float Z[3], A[3], B[3];          // offsets at the start poses
    unsigned short zab[10];          // their remainders (bfloat16)
    float E;                         // the error bound
    int body_a, body_b;
    unsigned key[2];                 // split keys of t | alpha << 16, beta (filter_split)
    unsigned lev;                    // first level within tolerance of t | alpha << 6 | beta << 12, flags
};
static_assert(sizeof(FilterRec) == 128, "one 128-byte line per candidate");
constexpr unsigned kRecFV = 1u << 18;       // face-vertex
constexpr unsigned kRecDouble = 1u << 19;   // searched in double alone
constexpr unsigned kRecShallow = 1u << 20;  // in double from time depth 7 on
// f stays within E on an axis: no box is surely a root, those within tolerance
// are decided in double where they are met; on two axes: next to none is dropped,
// the candidate is searched in double alone, from its seeds
constexpr unsigned kRecFlat = 1u << 21, kRecFlat2 = 1u << 22;

// candidate; index (24 bits) and level (5 bits) of time, alpha and beta
struct FNode {
    unsigned cand, x[3];
};
__device__ __forceinline__ int fn_level(const FNode& n, int d) { return (int)(n.x[d] >> 24); }
__device__ __forceinline__ unsigned fn_index(const FNode& n, int d) { return n.x[d] & 0xffffffu; }

struct FilterArgs {
    CCDArgs d;                       // the double-precision search's
    const FilterRec* rec;
    unsigned long long* state;       // per candidate
    const unsigned long long* flat;  // not 0: some candidates are flat
    const float* frames;             // nb x kTableSlots x kFrame32
    const float* bodies;             // nb x kBody32
    int64_t n;                       // candidates
    int seeds_log2;
    int window_log2;                 // first time window 2^-window_log2 (0: none)
    FNode* later;                    // gridDim x kFilterLists x later_cap boxes
    int later_cap;
    Piece* out;                      // pieces for the double-precision search
    unsigned long long* n_out;       // appended count (above cap: the call is redone without the filter)
    unsigned long long cap;
    unsigned long long* next;        // next batch of work items
    unsigned long long *boxes, *hits;
    unsigned long long* gmin;        // running minimum (double bits)
    unsigned long long* scene_gmin;  // batched contexts: the same per scene, else null
    const int* bscene;
};

// Coefficients of the k-th Taylor terms of S(s) = sin(sqrt s) / sqrt s =
// sum (-s)^j / (2j + 1)! and C(s) = (1 - cos(sqrt s)) / s =
// sum (-s)^j / (2j + 2)!: S^(k) / k! = sum_j binom(j, k) a_j s^(j - k)
struct SeriesTable {
    double a[2 * kTaylor][kSeries];
    constexpr SeriesTable() : a()
    {
        for (int f = 0; f < 2; f++)
            for (int k = 0; k < kTaylor; k++)
                for (int i = 0; i < kSeries; i++) {
                    const int j = i + k;
                    double v = j % 2 ? -1.0 : 1.0;
                    for (int q = 2; q <= 2 * j + 1 + f; q++) v /= q;
                    for (int q = 1; q <= k; q++) v = v * (j - k + q) / q;
                    a[f * kTaylor + k][i] = v;
                }
    }
};
__constant__ SeriesTable kSeriesTable = SeriesTable();

// One block per body: the start frame (R(theta0), p0) in double, deep_frame's
// data, and the table's frames relative to the start frame as middle and
// radius.  Bodies no candidate has may hold no frames in the table; theirs
// are not read.
__global__ void __launch_bounds__(kTableSlots)
k_filter_bodies(const double* __restrict__ table, const double* __restrict__ x0, const double* __restrict__ traj,
                double* __restrict__ ref, float* __restrict__ frames, float* __restrict__ bodies)
{
    __shared__ double base[kRef64];
    const int b = blockIdx.x, node = threadIdx.x;
    const double th[3] = { x0[6 * b + 3], x0[6 * b + 4], x0[6 * b + 5] };
    float* body = bodies + (size_t)b * kBody32;
    if (node == 0) {
        double R[9];
        rot_rn(th, R);
        for (int k = 0; k < 9; k++) base[k] = R[k];
        for (int k = 0; k < 3; k++) base[9 + k] = x0[6 * b + k];
        for (int k = 0; k < kRef64; k++) ref[(size_t)b * kRef64 + k] = base[k];
    } else if (node >= 32 && node < 32 + 2 * kTaylor) {
        const double s = th[0] * th[0] + th[1] * th[1] + th[2] * th[2];
        double v = 0.0;
        for (int i = kSeries - 1; i >= 0; i--) v = fma(v, s, kSeriesTable.a[node - 32][i]);
        body[9 + node - 32] = (float)v;
    } else if (node == 64) {
        // |dtheta| and |theta| over the step, rounded up
        float w2 = 0.0f, t2 = 0.0f;
        for (int k = 0; k < 3; k++) {
            const double* e = traj + (size_t)b * kTrajDoubles + 6;
            const float w = (float)(0.5 * (e[2 * (3 + k)] + e[2 * (3 + k) + 1]));
            body[k] = (float)th[k];
            body[3 + k] = w;
            body[6 + k] = (float)(0.5 * (e[2 * k] + e[2 * k + 1]));
            w2 = fmaf(w, w, w2);
            t2 = fmaf((float)th[k], (float)th[k], t2);
        }
        const float d = 1.001f * sqrtf(w2), r = 1.001f * sqrtf(t2) + d, sg = 2.0f * d * r;
        // out of the series' range: no deep frames (T = inf)
        const bool ok = sg <= 1.0f && r < kMaxTheta;
        body[21] = ok ? d + sg * (r * (1.0f / 6.0f) + 0.5f + r * r * (1.0f / 24.0f)) : INFINITY;
    }
    __syncthreads();
    const double* e = table + ((size_t)b * kTableSlots + node) * kTableEntry;
    float* o = frames + ((size_t)b * kTableSlots + node) * kFrame32;
    for (int k = 0; k < kRef64; k++) {
        const double lo = e[2 * k] - base[k], hi = e[2 * k + 1] - base[k];
        const int at = k < 9 ? k : 18 + (k - 9), rad = k < 9 ? 9 : 3;
        o[at] = (float)(0.5 * (lo + hi));
        o[at + rad] = __double2float_ru(0.5 * (hi - lo));
    }
}

struct F2 {
    float lo, hi;
};

// bounds of x y - x0 y0 over x = x0 + dx, y = y0 + dy: x0 dy + dx (y0 + dy)
// at the four corners
__device__ __forceinline__ F2 prod_diff(float x0, F2 dx, float y0, F2 dy)
{
    const float yl = y0 + dy.lo, yh = y0 + dy.hi, ql = x0 * dy.lo, qh = x0 * dy.hi;
    const float a = fmaf(dx.lo, yl, ql), b = fmaf(dx.lo, yh, qh), c = fmaf(dx.hi, yl, ql), d = fmaf(dx.hi, yh, qh);
    return F2 { fminf(fminf(a, b), fminf(c, d)), fmaxf(fmaxf(a, b), fmaxf(c, d)) };
}

__device__ __forceinline__ float taylor_diff(const float* c, float d)
{
    float v = c[kTaylor - 1];
#pragma unroll
    for (int k = kTaylor - 2; k >= 1; k--) v = fmaf(v, d, c[k]);
    return v * d;
}

// The interval frame of a body over [t0, t1] minus its start frame, from the
// expressions of body_at and irotation written as differences from t = 0, so
// that every rounding is relative to a difference.  With theta = theta0 +
// dtheta t, s = |theta|^2, the interval rotation is I + S(s) K + C(s) K^2
// (S = sinc|theta|, C = sinc(|theta|/2)^2 / 2, both decreasing for |theta| <
// 4.49, so the interval's ends give their bounds), K^2's entries sums of the
// products theta_i theta_j bounded as independent factors.  The ends of S and
// C come from six terms about s0 (remainder below 1.6e-10 |ds|^6, |ds| <= 1).
// Errors, with d = |dtheta|, r = |theta0| + d, sg = 2 d r >= |ds| and every
// |theta_i theta_j| difference: theta 2 u d; ds 8 u sg; S 14 u sg / 6; S K
// 5 u d + 18 u sg r / 6; K^2 8 u sg; C 14 u sg / 24; C K^2 6 u sg +
// 18 u sg r^2 / 24; the entry 20 u T with T = d + sg (r / 6 + 1 / 2 + r^2 / 24).
__device__ __forceinline__ void deep_frame(const float* __restrict__ body, float t0, float t1, float f[kFrame32])
{
    const float4* p = reinterpret_cast<const float4*>(body);
    float g[kBody32];
#pragma unroll
    for (int k = 0; k < kBody32 / 4; k++) {
        const float4 x = __ldg(p + k);
        g[4 * k] = x.x;
        g[4 * k + 1] = x.y;
        g[4 * k + 2] = x.z;
        g[4 * k + 3] = x.w;
    }
    const float *th = g, *S = g + 9, *C = g + 15;
    F2 D[3], q[3], ds { 0.0f, 0.0f };
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float a = g[3 + k] * t0, b = g[3 + k] * t1;
        D[k] = F2 { fminf(a, b), fmaxf(a, b) };
        const float rl = th[k] + D[k].lo, rh = th[k] + D[k].hi;
        const float ll = D[k].lo * (th[k] + rl), hh = D[k].hi * (th[k] + rh);
        const float lh = fmaf(D[k].lo, rh, th[k] * D[k].hi);
        const float mn = fminf(ll, hh), mx = fmaxf(ll, hh);
        // |theta_k|^2 as an interval starts at 0 when theta_k changes sign
        ds.lo += rl < 0.0f && rh > 0.0f ? -th[k] * th[k] : mn;
        ds.hi += mx;
        q[k] = F2 { fminf(mn, lh), fmaxf(mx, lh) };
        const float pa = g[6 + k] * t0, pb = g[6 + k] * t1;
        f[18 + k] = 0.5f * (pa + pb);
        f[21 + k] = 0.5f * fabsf(pb - pa);
    }
    const F2 dS { taylor_diff(S, ds.hi), taylor_diff(S, ds.lo) }, dC { taylor_diff(C, ds.hi), taylor_diff(C, ds.lo) };
    F2 A[3];
#pragma unroll
    for (int k = 0; k < 3; k++) A[k] = prod_diff(S[0], dS, th[k], D[k]);
    auto put = [&](int i, float lo, float hi) {
        f[i] = 0.5f * (lo + hi);
        f[9 + i] = 0.5f * (hi - lo);
    };
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int j = (i + 1) % 3, k = (i + 2) % 3;
        // diagonal: -(theta_j^2 + theta_k^2)
        const F2 n = prod_diff(C[0], dC, -(th[j] * th[j] + th[k] * th[k]), F2 { -(q[j].hi + q[k].hi), -(q[j].lo + q[k].lo) });
        put(4 * i, n.lo, n.hi);
        // the pair (j, k), its K entry -+theta_i: K_jk = -theta_i, K_kj = theta_i
        const F2 m = prod_diff(C[0], dC, th[j] * th[k], prod_diff(th[j], D[j], th[k], D[k]));
        put(3 * j + k, m.lo - A[i].hi, m.hi - A[i].lo);
        put(3 * k + j, m.lo + A[i].lo, m.hi + A[i].hi);
    }
}

// a double as a float and a bfloat16 remainder
__device__ __forceinline__ float split_pair(double x, unsigned short& rest)
{
    const float h = (float)x;
    rest = __bfloat16_as_ushort(__float2bfloat16_rn((float)(x - (double)h)));
    return h;
}
__device__ __forceinline__ float pair_rest(unsigned short b) { return __uint_as_float((unsigned)b << 16); }

// bound of the displacements along axis c over [0, 1] (rarely asked for)
static __device__ __noinline__ float filter_axis_motion(const FilterRec& r, const Query& q,
                                                        const float* __restrict__ frames, int c)
{
    float D = 0.0f;
    for (int v = 0; v < 4; v++) {
        const float* root = frames + (size_t)(v < (q.fv ? 1 : 2) ? q.body_a : q.body_b) * kTableSlots * kFrame32;
        float d = fabsf(root[18 + c]) + root[21 + c];
        for (int k = 0; k < 3; k++) d = fmaf(fabsf(r.v[v][k]), fabsf(root[3 * c + k]) + root[9 + 3 * c + k], d);
        D = fmaxf(D, d);
    }
    return D;
}

// the record of a candidate (rest vertices and bodies in q) without its
// tolerances' part
__device__ __forceinline__ void filter_record(const Query& q, const double* __restrict__ ref,
                                              const float* __restrict__ frames,
                                              const float* __restrict__ bodies, FilterRec& r)
{
    const int na = q.fv ? 1 : 2;
    double X[4][3];
    float D = 0.0f, W = 0.0f, Tv = 0.0f, m = 0.0f;
    float all = 0.0f;  // NaN when a position or displacement is (the maxima pass over NaN)
    const float Ta = bodies[(size_t)q.body_a * kBody32 + 21], Tb = bodies[(size_t)q.body_b * kBody32 + 21];
    const bool deep = Ta < INFINITY && Tb < INFINITY;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int b = v < na ? q.body_a : q.body_b;
        const double* R = ref + (size_t)b * kRef64;
        const float* root = frames + (size_t)b * kTableSlots * kFrame32;
        float l1 = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            r.v[v][k] = (float)q.v[v][k];
            l1 += fabsf(r.v[v][k]);
        }
        if (deep) Tv = fmaxf(Tv, l1 * (v < na ? Ta : Tb));
        W = fmaxf(W, l1);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            X[v][c] = fma(q.v[v][2], R[3 * c + 2], fma(q.v[v][1], R[3 * c + 1], fma(q.v[v][0], R[3 * c], R[9 + c])));
            float d = fabsf(root[18 + c]) + root[21 + c];
#pragma unroll
            for (int k = 0; k < 3; k++)
                d = fmaf(fabsf(r.v[v][k]), fabsf(root[3 * c + k]) + root[9 + 3 * c + k], d);
            D = fmaxf(D, d);
            W = fmaxf(W, fabsf((float)X[v][c]));
            all += 0.0f * (d + (float)X[v][c]);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        r.Z[c] = split_pair(X[0][c] - (q.fv ? X[1][c] : X[2][c]), r.zab[c]);
        r.A[c] = split_pair((q.fv ? X[2][c] : X[0][c]) - X[1][c], r.zab[3 + c]);
        r.B[c] = split_pair(X[3][c] - (q.fv ? X[1][c] : X[2][c]), r.zab[6 + c]);
        m = fmaxf(m, fmaxf(fabsf(r.Z[c]), fmaxf(fabsf(r.A[c]), fabsf(r.B[c]))));
    }
    r.zab[9] = 0;
    // 1.01: this bound's own rounding; W: positions and |v| of every term
    const float u = 5.9604644775390625e-08f;
    r.E = 1.01f * (96.0f * u * D + 120.0f * u * Tv + 9.313225746154785e-10f * m + 1.1368683772161603e-13f * (W + D));
    r.body_a = q.body_a;
    r.body_b = q.body_b;
    r.lev = (q.fv ? kRecFV : 0u) | (deep ? 0u : kRecShallow);
    int flat = 0;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float w = fabsf(r.Z[c]) + fabsf(r.A[c]) + fabsf(r.B[c]);
        if (w <= r.E && w + 6.0f * filter_axis_motion(r, q, frames, c) <= r.E) flat++;
    }
    r.lev |= (flat > 0 ? kRecFlat : 0u) | (flat > 1 ? kRecFlat2 : 0u);
    // finite bounds and tolerances whose keys order the splits; anything
    // else is left to the double-precision search from its root
    if (!(r.E < 1e18f) || !(m < 1e18f) || !(all == 0.0f)) r.lev |= kRecDouble;
}

// the tolerances' part
__device__ __forceinline__ void filter_levels(const double tol[3], FilterRec& r)
{
    const TolKeys K = tol_keys(tol);
    unsigned lev = r.lev;
    if (!K.ok) lev |= kRecDouble;
    // K[d] + lv[d] 2^52 (split_dim_keys) in the order of its exponent plus
    // level, then its mantissa: 4 exponent + the mantissa's rank
    unsigned key[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        unsigned rank = 0;
#pragma unroll
        for (int o = 0; o < 3; o++)
            rank += (K.tk[o] & 0xfffffffffffffll) < (K.tk[d] & 0xfffffffffffffll) ? 1u : 0u;
        key[d] = (unsigned)((K.tk[d] >> 52) & 0x7ff) << 2 | rank;
        // first level l with (1 + 2^-52) 2^-l <= tol (node_widths)
        int l = 0;
        while (l < 63 && !le_nn(__longlong_as_double(((long long)(1023 - l) << 52) + 1ll), tol[d])) l++;
        lev |= (unsigned)l << (6 * d);
    }
    r.key[0] = key[0] | key[1] << 16;
    r.key[1] = key[2];
    r.lev = lev;
}

// bounds of a vertex's displacement
__device__ __forceinline__ void filter_vertex(const float* f, const float v[3], float lo[3], float hi[3])
{
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float m = fmaf(v[2], f[3 * c + 2], fmaf(v[1], f[3 * c + 1], fmaf(v[0], f[3 * c], f[18 + c])));
        const float r = fmaf(fabsf(v[2]), f[9 + 3 * c + 2],
                             fmaf(fabsf(v[1]), f[9 + 3 * c + 1], fmaf(fabsf(v[0]), f[9 + 3 * c], f[21 + c])));
        lo[c] = m - r;
        hi[c] = m + r;
    }
}

// The bounds of y over [0, toi_tol] and the tolerances' boxes of alpha and beta
// exclude zero on an axis, in double too: |y - Z| is at most the displacements
// over [0, toi_tol] (the table's last slot), A and B and twice the displacements
// times the widths, and E covers the rest as for any box.
__device__ __forceinline__ bool filter_starts_apart(const FilterRec& r, const float* __restrict__ frames,
                                                    float w1, float w2)
{
    if (r.lev & kRecDouble) return false;
    float d[3] = { 0.0f, 0.0f, 0.0f };
    const int na = r.lev & kRecFV ? 1 : 2;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const float* f = frames + ((size_t)(v < na ? r.body_a : r.body_b) * kTableSlots + kTableNodes) * kFrame32;
        float lo[3], hi[3];
        filter_vertex(f, r.v[v], lo, hi);
#pragma unroll
        for (int c = 0; c < 3; c++) d[c] = fmaxf(d[c], fmaxf(fabsf(lo[c]), fabsf(hi[c])));
    }
    bool apart = false;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float w = 2.0f * d[c] + w1 * (fabsf(r.A[c]) + 2.0f * d[c]) + w2 * (fabsf(r.B[c]) + 2.0f * d[c]);
        apart = apart || fabsf(r.Z[c]) > 1.001f * (w + r.E);
    }
    return apart;
}

__device__ __forceinline__ void filter_frame(const float* __restrict__ g, float f[kFrame32])
{
    const float4* p = reinterpret_cast<const float4*>(g);
#pragma unroll
    for (int k = 0; k < kFrame32 / 4; k++) {
        const float4 x = __ldg(p + k);
        f[4 * k] = x.x;
        f[4 * k + 1] = x.y;
        f[4 * k + 2] = x.z;
        f[4 * k + 3] = x.w;
    }
}

// a + b exactly as s + e
__device__ __forceinline__ float two_sum(float a, float b, float& e)
{
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
    return s;
}

// Whether the double-precision bounds of f over the box exclude zero (-1),
// include it (1), or cannot be told (0).  slot < 0: frames from deep_frame.
// The box starts at (a0, b0) with widths wa, wb.
__device__ __forceinline__ int filter_test(const FilterRec& r, bool fv, const float* __restrict__ frames,
                                           const float* __restrict__ bodies, int slot, float t0, float t1,
                                           float a0, float wa, float b0, float wb)
{
    float lo[4][3], hi[4][3];
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const int b = side ? r.body_b : r.body_a;
        float f[kFrame32];
        if (slot >= 0) filter_frame(frames + ((size_t)b * kTableSlots + slot) * kFrame32, f);
        else deep_frame(bodies + (size_t)b * kBody32, t0, t1, f);
        if (side == 0) filter_vertex(f, r.v[0], lo[0], hi[0]);
        if ((side == 1) == fv) filter_vertex(f, r.v[1], lo[1], hi[1]);
        if (side == 1) filter_vertex(f, r.v[2], lo[2], hi[2]);
        if (side == 1) filter_vertex(f, r.v[3], lo[3], hi[3]);
    }
    const float a1 = a0 + wa, b1 = b0 + wb;  // exact
    bool out = false, in = true;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        // Z - A a0 - B b0 as base + rest
        const float A = r.A[c], B = r.B[c];
        const float pa = __fmul_rn(A, a0), pb = __fmul_rn(B, b0);
        float ea, eb;
        const float s1 = two_sum(r.Z[c], -pa, ea), base = two_sum(s1, -pb, eb);
        const float rest = (ea + eb) - __fmaf_rn(A, a0, -pa) - __fmaf_rn(B, b0, -pb)
            + (pair_rest(r.zab[c]) - pair_rest(r.zab[3 + c]) * a0 - pair_rest(r.zab[6 + c]) * b0);
        const float kl = fv ? lo[1][c] : lo[2][c], kh = fv ? hi[1][c] : hi[2][c];
        const float Fl = (fv ? lo[2][c] : lo[0][c]) - hi[1][c], Fh = (fv ? hi[2][c] : hi[0][c]) - lo[1][c];
        const float Gl = lo[3][c] - kh, Gh = hi[3][c] - kl;
        const float Aw = A * wa, Bw = B * wb;
        const float l = (lo[0][c] - kh) - fmaxf(Fh * a0, fmaf(Fh, a1, Aw)) - fmaxf(Gh * b0, fmaf(Gh, b1, Bw));
        const float h = (hi[0][c] - kl) - fminf(Fl * a0, fmaf(Fl, a1, Aw)) - fminf(Gl * b0, fmaf(Gl, b1, Bw));
        const float yl = (base + l) + rest, yh = (base + h) + rest;
        const float E = fmaf(fabsf(Aw) + fabsf(Bw), 4.76837158203125e-07f, r.E);
        out = out || yl > E || yh < -E;
        in = in && yl <= -E && yh >= E;
    }
    return out ? -1 : in ? 1 : 0;
}

// The dimension a node splits: the smallest key plus level among the
// dimensions above tolerance (split_dim_keys); -1 when there is none
__device__ __forceinline__ int filter_split(const FilterRec& r, const FNode& x)
{
    const unsigned key[3] = { r.key[0] & 0xffffu, r.key[0] >> 16, r.key[1] };
    int s = -1;
    unsigned ks = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const unsigned lv = (unsigned)fn_level(x, d), kd = key[d] + 4u * lv;
        if (lv < ((r.lev >> (6 * d)) & 63u) && (s < 0 || kd < ks)) {
            s = d;
            ks = kd;
        }
    }
    return s;
}

// the half of a node along dimension s
__device__ __forceinline__ FNode filter_half(FNode x, int s, unsigned upper)
{
#pragma unroll
    for (int d = 0; d < 3; d++)
        if (d == s) x.x[d] = (x.x[d] & 0xff000000u) + (1u << 24) + (2u * fn_index(x, d) | upper);
    return x;
}

// the list of a box starting at time index it of level lt: -1 before the
// first window 2^-k, else the power of two below its start, from 2^-k on
__device__ __forceinline__ int filter_list(unsigned it, int lt, int k)
{
    const int e = (31 - __clz((int)it)) - lt + k;  // it = 0: the clz is 32
    return it == 0 || k == 0 || e < 0 ? -1 : min(e, kFilterLists - 1);
}

// a box of a later window than the one searched goes to its list, while
// there is room (the counts of full lists are clamped after the block's next
// barrier); false: it is searched now
__device__ __forceinline__ bool filter_defer(const FilterArgs& a, FNode* later, int* later_cnt, int cur,
                                             const FNode& x)
{
    const int l = filter_list(fn_index(x, 0), fn_level(x, 0), a.window_log2);
    if (l <= cur) return false;
    const int o = atomicAdd(&later_cnt[l], 1);
    if (o >= a.later_cap) return false;
    later[(size_t)l * a.later_cap + o] = x;
    return true;
}

// Node j at depth seeds_log2 of a candidate's tree (seed_node); a candidate
// left to the double-precision search, or within tolerance above that depth,
// has one for all j below its node: false for the others
__device__ __forceinline__ bool filter_seed(const FilterRec& r, int seeds_log2, unsigned j, FNode& x)
{
    int l = seeds_log2 - 1;
    for (; l >= 0; l--) {
        const int s = (r.lev & kRecDouble) ? -1 : filter_split(r, x);
        if (s < 0) break;
        x = filter_half(x, s, (j >> l) & 1u);
    }
    return l < 0 || (j & ((2u << l) - 1u)) == 0;
}

// (its budget starts with the boxes on its path)
__device__ __forceinline__ Piece filter_piece(const FNode& x)
{
    Piece pc;
    pc.cand = x.cand;
    pc.earliest = INFINITY;
    pc.depth = 0;
    for (int d = 0; d < 3; d++) {
        pc.ix[d] = fn_index(x, d);
        pc.lv[d] = fn_level(x, d);
        pc.depth += pc.lv[d];
    }
    pc.boxes = (unsigned long long)pc.depth;
    return pc;
}

// f_zero of a box in double precision
static __device__ __noinline__ bool filter_exact(const CCDArgs& a, const FNode& x)
{
    Query q;
    load_candidate(a, x.cand, q);
    Node n { { 0, 0, 0 }, { 0ull, 0ull, 0ull }, 0 };
    for (int d = 0; d < 3; d++) {
        n.lv[d] = fn_level(x, d);
        n.ix[d] = fn_index(x, d);
    }
    const Box b = node_box(n);
    const int na = q.fv ? 1 : 2;
    Itv R[9], p[3];
    frame_compute(a, q.body_a, Itv { b.t0, b.t1 }, R, p);
    for (int v = 0; v < na; v++) iworld_vertex(R, p, q.v[v], q.P[v]);
    frame_compute(a, q.body_b, Itv { b.t0, b.t1 }, R, p);
    for (int v = na; v < 4; v++) iworld_vertex(R, p, q.v[v], q.P[v]);
    return f_zero(q, b);
}

// one more undecided box of a candidate (weight k): its state
__device__ __forceinline__ unsigned long long filter_undecided(const FilterArgs& a, unsigned cand, unsigned k)
{
    return atomicAdd(a.state + cand, (unsigned long long)k << 32) + ((unsigned long long)k << 32);
}
__device__ __forceinline__ bool past_limit(unsigned long long state)
{
    return (unsigned)((state & ~kHandedOn) >> 32) >= kUndecidedLimit;
}

__device__ __forceinline__ void record_root(const FilterArgs& a, const FNode& x)
{
    const unsigned long long t0 = (unsigned long long)dbits(dyadic(fn_index(x, 0), fn_level(x, 0)));
    atomicMin(a.gmin, t0);
    if (a.scene_gmin) atomicMin(a.scene_gmin + a.bscene[a.rec[x.cand].body_a], t0);
}

// A candidate is handed on: its seeds as pieces (told from its earlier ones by 0
// boxes), once; false: they did not fit
static __device__ __noinline__ bool filter_hand_on(const FilterArgs& a, unsigned cand)
{
    if (atomicOr(a.state + cand, kHandedOn) & kHandedOn) return true;
    const unsigned n = 1u << a.seeds_log2;
    const unsigned long long o = atomicAdd(a.n_out, (unsigned long long)n);
    if (o + n > a.cap) return false;
    for (unsigned j = 0; j < n; j++) {
        FNode x { cand, { 0, 0, 0 } };
        const bool own = filter_seed(a.rec[cand], a.seeds_log2, j, x);
        Piece pc = filter_piece(x);
        pc.boxes = 0;
        if (!own) pc.cand = -1;
        a.out[o + j] = pc;
    }
    return true;
}

// kExact: for calls with flat candidates, whose boxes within tolerance are
// decided here, in double, so that the running minimum falls in this launch (a
// slab of 36 x 36 quads landing on another, aligned: 14.9 -> 1.4 ms).  It is done between the turns, which the call would otherwise cost
// registers (a 200-link chain in line, without a box to decide, 1.40 -> 1.54 ms;
// so 1.45); both are launched, and the wrong one ends at once.
template <bool kExact>
__global__ void __launch_bounds__(kFilterThreads, kFilterBlocks)
k_ccd_filter(FilterArgs a)
{
    if ((*a.flat != 0) != kExact) return;
    __shared__ FNode stack[kFilterStack];
    __shared__ int pushes[2][kFilterThreads / 32];  // per warp: lower halves | upper halves << 16
    __shared__ int later_cnt[kFilterLists];
    __shared__ unsigned long long batch, gmin_seen;
    __shared__ bool full, over;      // the pieces have run over their buffer: seen by this block, by any
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    FNode* later = a.later + (size_t)blockIdx.x * kFilterLists * a.later_cap;
    const unsigned long long nwork = (unsigned long long)a.n << a.seeds_log2;
    // the work items of a batch come from distant places of the list, so that
    // neighbouring candidates (of one contact) spread over the blocks
    const unsigned long long batches = (nwork + kFilterThreads - 1) / kFilterThreads;
    unsigned long long tot = 0, hits = 0;
    bool more = true;
    int cnt = 0;                     // pending boxes (the same in every thread)
    int cur = -1;                    // the list being searched
    // kExact: the turns stop when boxes are to be decided in double (a call
    // within them would cost every turn its registers)
    __shared__ FNode exact_box[kExact ? kFilterThreads : 1];
    __shared__ int n_exact;
    __shared__ bool exact_full;
    bool pause = false;
    int turn = 0;
    if (tid < kFilterLists) later_cnt[tid] = 0;
    if (tid == 0) {
        full = exact_full = false;
        n_exact = 0;
    }
    __syncthreads();
    do {
        pause = false;
        for (;; turn ^= 1) {
            bool mine = false;
            FNode x { 0, { 0, 0, 0 } };
            if (cnt < kFilterThreads / 2 && more) {
                // a batch of new work items, one per thread, and nothing from the stack
                if (tid == 0) {
                    batch = atomicAdd(a.next, 1ull);
                    over = *(volatile unsigned long long*)a.n_out > a.cap;
                }
                __syncthreads();
                unsigned long long w = batch;
                const bool stop = over;
                __syncthreads();
                if (stop) break;
                if (w >= batches) {
                    more = false;
                    continue;
                }
                w += (unsigned long long)tid * batches;
                if (w < nwork) {
                    x.cand = (unsigned)(w % (unsigned long long)a.n);
                    mine = filter_seed(a.rec[x.cand], a.seeds_log2, (unsigned)(w / (unsigned long long)a.n), x);
                }
            } else if (cnt > 0) {
                const int n = min(cnt, kFilterThreads);
                mine = tid < n;
                if (mine) x = stack[cnt - 1 - tid];
                cnt -= n;
            } else {
                // the next list; a list after a single scene's first impact and
                // all later ones are dropped
                if (cur >= 0) {
                    const int left = later_cnt[cur];
                    __syncthreads();
                    if (left > 0) {
                        const int n = min(left, kFilterThreads);
                        mine = tid < n;
                        if (mine) x = later[(size_t)cur * a.later_cap + left - 1 - tid];
                        if (tid == 0) later_cnt[cur] = left - n;
                    }
                    if (left == 0) {
                        if (++cur >= kFilterLists) break;
                        continue;
                    }
                } else {
                    cur = 0;
                    continue;
                }
                if (!a.scene_gmin) {
                    if (tid == 0) gmin_seen = *(volatile unsigned long long*)a.gmin;
                    __syncthreads();
                    if (gmin_seen <= (unsigned long long)(1023 + cur - a.window_log2) << 52) break;
                }
            }
            const int lt = fn_level(x, 0), la = fn_level(x, 1), lb = fn_level(x, 2);
            const unsigned it = fn_index(x, 0), ia = fn_index(x, 1), ib = fn_index(x, 2);
            bool emit = false, split = false, low = false, hand_on = false, exact = false;
            int s = 0;
            FNode up = x;                // the upper half
            bool high = false;
            if (mine) {
                const unsigned long long t0 = (unsigned long long)dbits(dyadic(it, lt));
                // integers on 2^-24: a0 + b0 <= 1 (add_dn rounds exact sums, so
                // its test is this one), and the upper sum is never negative
                const unsigned fa = ia << (kFilterLevel - la), fb = ib << (kFilterLevel - lb);
                const FilterRec& r = a.rec[x.cand];
                const unsigned lev = r.lev;
                const bool fv = (lev & kRecFV) != 0, searched = !(lev & (kRecDouble | kRecFlat2));
                unsigned long long* g = a.scene_gmin ? a.scene_gmin + a.bscene[r.body_a] : a.gmin;
                bool keep = t0 < *(volatile unsigned long long*)g && !(fv && fa + fb > (1u << kFilterLevel));
                // a seed of a later window, or a box its list had no room for
                if (keep) keep = !filter_defer(a, later, later_cnt, cur, x);
                if (keep) {
                    // exact: integers up to 2^24 times a power of two
                    const float wt = __int_as_float((127 - lt) << 23);
                    const float wa = __int_as_float((127 - la) << 23), wb = __int_as_float((127 - lb) << 23);
                    tot++;
                    int in = 0;
                    s = -1;
                    unsigned long long seen = 0;
                    if (searched) {
                        // (every fourth level: the memory's latency is 2 % of a call)
                        if ((lt + la + lb) % 4 == 0) seen = *(volatile unsigned long long*)(a.state + x.cand);
                        in = filter_test(r, fv, a.frames, a.bodies, lt < kTableDepth ? (1 << lt) - 1 + (int)it : -1,
                                         (float)it * wt, (float)(it + 1) * wt, (float)ia * wa, wa, (float)ib * wb, wb);
                        s = filter_split(r, x);
                    }
                    if (seen & kHandedOn) in = -1;
                    if (in >= 0) {
                        // split: not within tolerance, and the halves have frames
                        // and exact levels
                        const int limit = s == 0 && (lev & kRecShallow) ? kTableDepth - 1 : kFilterLevel - 1;
                        split = s >= 0 && (s == 0 ? lt : s == 1 ? la : lb) < limit;
                        if (split) {
                            low = high = true;
                            up = filter_half(x, s, 1u);
                        } else if (s < 0 && in > 0 && it > 0) {
                            // a root: within tolerance, after t = 0, zero inside
                            record_root(a, x);
                            hits++;
                        } else {
                            // (a flat candidate's boxes within tolerance are decided below)
                            exact = kExact && searched && s < 0 && it > 0 && (lev & kRecFlat);
                            if (!exact) {
                                emit = true;
                                if (searched) {
                                    const unsigned long long u = filter_undecided(a, x.cand, s < 0 ? kUndecidedLeaf : 1u);
                                    emit = !(u & kHandedOn);
                                    hand_on = past_limit(u);
                                }
                            }
                        }
                    }
                }
                if (high) high = !filter_defer(a, later, later_cnt, cur, up);
            }
            // halves: the lower ones on top; without room the box itself goes on
            const unsigned ml = __ballot_sync(0xffffffffu, low), mh = __ballot_sync(0xffffffffu, high);
            if (lane == 0) pushes[turn][warp] = __popc(ml) | __popc(mh) << 16;
            __syncthreads();             // the boxes popped are read, the counts written
            if (tid < kFilterLists && later_cnt[tid] > a.later_cap) later_cnt[tid] = a.later_cap;
            int all = 0, before = 0;
#pragma unroll
            for (int k = 0; k < kFilterThreads / 32; k++) {
                const int q = pushes[turn][k];
                all += q;
                if (k < warp) before += q;
            }
            const int nl = all & 0xffff, nh = all >> 16;
            if (cnt + nl + nh > kFilterStack) {
                // (counted: a search that fills the stack without deciding is handed on)
                if (split) {
                    const unsigned long long u = filter_undecided(a, x.cand, 1u);
                    emit = !(u & kHandedOn);
                    hand_on = past_limit(u);
                }
            } else {
                if (high) stack[cnt + nh - 1 - (before >> 16) - __popc(mh & below)] = up;
                if (low) stack[cnt + nh + nl - 1 - (before & 0xffff) - __popc(ml & below)] = filter_half(x, s, 0u);
                cnt += nl + nh;
            }
            if (kExact && exact) exact_box[atomicAdd(&n_exact, 1)] = x;
            const unsigned e = __ballot_sync(0xffffffffu, emit);
            if (e) {
                unsigned long long o = 0;
                if (lane == 0) o = atomicAdd(a.n_out, (unsigned long long)__popc(e));
                o = __shfl_sync(0xffffffffu, o, 0) + __popc(e & below);
                if (emit && o < a.cap) a.out[o] = filter_piece(x);
                if (emit && o >= a.cap) full = true;
            }
            if (hand_on && !filter_hand_on(a, x.cand)) full = true;
            __syncthreads();             // the pushed boxes and full are written
            if (full) break;
            if (kExact && n_exact > 0) {
                pause = true;
                break;
            }
        }
        if (kExact && pause) {
            if (tid < n_exact) {
                const FNode x = exact_box[tid];
                if (filter_exact(a.d, x)) {
                    record_root(a, x);
                    hits++;
                } else if (past_limit(filter_undecided(a, x.cand, kUndecidedLeaf)) && !filter_hand_on(a, x.cand)) {
                    exact_full = true;
                }
            }
            __syncthreads();             // the boxes are read, exact_full is written
            if (tid == 0) n_exact = 0;
            pause = !exact_full;
        }
    } while (kExact && pause);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tot += __shfl_down_sync(0xffffffffu, tot, o);
        hits += __shfl_down_sync(0xffffffffu, hits, o);
    }
    if (lane == 0 && tot) atomicAdd(a.boxes, tot);
    if (lane == 0 && hits) atomicAdd(a.hits, hits);
}

} // namespace rigc

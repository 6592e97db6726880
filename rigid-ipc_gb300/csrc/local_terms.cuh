// Device helpers shared by the per-constraint local terms (barrier and
// friction): vertex positions with their rotation derivatives, body-space
// images of vertex-space vectors, shared-memory Hessian accumulators, the
// rigid curvature term of apply_chain_rule
// (src/problems/distance_barrier_rb_problem.cpp:1182-1248) and the PSD
// projection.
//
// A constraint's energy depends on its bodies' translations through their
// difference t_a - t_b only, so its 12x12 Hessian over (t_a, theta_a, t_b,
// theta_b) is that over (t_a, theta_a, theta_b) with the rows and columns of
// t_b the negatives of t_a's.  The kernels accumulate those 9 rows (45
// entries).  In the orthonormal basis with (t_a - t_b) / sqrt 2 in the place
// of the translations the Hessian is the 9x9 with its t_a rows and columns
// times sqrt 2 (and zero on t_a + t_b), so the projection is that of the 9x9.
#pragma once

#include "common.cuh"
#include "rotation.cuh"

namespace rigc {

// ---------------------------------------------------------------------------

constexpr int kBarrierTPB = 32;

struct Vtx {
    double X[3];     // world position
    double D[3][3];  // dX/dtheta  [coord][k]
};

__device__ __forceinline__ void cross(const double* a, const double* b, double* r)
{
    r[0] = a[1] * b[2] - a[2] * b[1];
    r[1] = a[2] * b[0] - a[0] * b[2];
    r[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ double dot(const double* a, const double* b)
{
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// reduced index (t_a 0-2, theta_a 3-5, theta_b 6-8) of body lb's rotation
__device__ __forceinline__ int red_rot(int lb) { return 3 + 3 * lb; }

// shared-memory symmetric 9x9 of one constraint: element (r, c), r >= c, in
// the lower triangle of a full row-major 9x9 whose entries are `stride`
// doubles apart (the constraints of a warp interleaved, the stride odd so that
// both a warp over constraints and a warp over entries meet all banks)
constexpr int kRed = 9;
struct SMat {
    double* base;
    int stride;
    __device__ __forceinline__ double& full(int r, int c) const { return base[(r * kRed + c) * stride]; }
    // entry (r, c) of the upper triangle, r <= c
    __device__ __forceinline__ double& at(int r, int c) const { return full(c, r); }
    __device__ __forceinline__ void clear() const
    {
        for (int r = 0; r < kRed; r++)
            for (int c = 0; c <= r; c++) full(r, c) = 0;
    }
};

// the reduced entries of a body-space 12-vector
__device__ __forceinline__ void reduce12(const double* g, double* r)
{
#pragma unroll
    for (int k = 0; k < 6; k++) r[k] = g[k];
#pragma unroll
    for (int k = 6; k < 9; k++) r[k] = g[k + 3];
}

// H += a00 v0 v0^T + a01 (v0 v1^T + v1 v0^T) + a11 v1 v1^T (v0, v1 reduced).
// The order of the two products is no more accurate than the other: with this one
// the converged run of 27 landing cubes (test_gpu_step.py; one of its steps has
// outcomes 2e-8 apart) ends at an outcome that the oracle has, with the other at a
// third, 1.02e-8 from the nearest.
__device__ __forceinline__ void add_quadratic(SMat H, double a00, double a01, double a11, const double* v0,
                                              const double* v1)
{
    for (int r = 0; r < kRed; r++) {
        const double u0 = a00 * v0[r] + a01 * v1[r], u1 = a01 * v0[r] + a11 * v1[r];
        for (int c = r; c < kRed; c++) H.at(r, c) += u1 * v1[c] + u0 * v0[c];
    }
}

// body-space image of a per-vertex vector field: out[6 lb + 0..2] += g_i,
// out[6 lb + 3 + k] += D_i[:, k] . g_i
__device__ __forceinline__ void to_body(const Vtx* V, const int* lbody, int nvc,
                                        const double (*g)[3], double* out)
{
    for (int k = 0; k < 12; k++) out[k] = 0;
    for (int i = 0; i < nvc; i++) {
        int o = 6 * lbody[i];
        for (int j = 0; j < 3; j++) out[o + j] += g[i][j];
        for (int k = 0; k < 3; k++)
            out[o + 3 + k] += V[i].D[0][k] * g[i][0] + V[i].D[1][k] * g[i][1] + V[i].D[2][k] * g[i][2];
    }
}

// curvature term: H(rot lb, rot lb) += sum_i g_i . (d2R_kl v_i) over the
// vertices i of each body, as d2R_kl : (sum_i g_i v_i^T)
__device__ __forceinline__ void add_curvature(SMat H, const double* const* frames, const int* lbody, int nvc,
                                              const double (*v)[3], const double (*g)[3])
{
    for (int b = 0; b < 2; b++) {
        double S[9];
        for (int k = 0; k < 9; k++) S[k] = 0;
        for (int i = 0; i < nvc; i++)
            if (lbody[i] == b)
                for (int j = 0; j < 3; j++)
                    for (int c = 0; c < 3; c++) S[3 * j + c] += g[i][j] * v[i][c];
        const double* d2 = frames[b] + 36;
        const int o = red_rot(b);
        for (int k = 0; k < 3; k++)
            for (int l = k; l < 3; l++) {
                const double* M = d2 + 9 * sym_index(k, l);
                double acc = 0;
                for (int e = 0; e < 9; e++) acc += M[e] * S[e];
                H.at(o + k, o + l) += acc;
            }
    }
}

// ---------------------------------------------------------------------------
// PSD projection of one 9x9 (lower triangle filled): A + V max(-L, 0) V^T from
// the eigen-decomposition A = V L V^T (as project_to_psd does, a matrix with
// no negative eigenvalue is left as it is), by Householder tridiagonalisation and the
// implicit symmetric QR algorithm with Wilkinson shifts (Golub & Van Loan,
// Matrix Computations, algorithms 8.3.1 - 8.3.3), in double throughout.
//
// W lanes share one matrix, each taking every W-th row (or column): W = 1 for
// many constraints (a thread per constraint: every FP64 instruction of a warp
// works on 32 matrices; an FP64 warp instruction takes this GPU's FP64 unit 64
// cycles whatever its active lanes), more for few (a shorter chain per
// matrix).  Every W computes each number by the same operations in the same
// order (products that feed sums are rounded explicitly, so that no
// instantiation contracts them), so the results are the same bits.  The scalars of a step (rotations,
// shifts, the tridiagonal matrix) are computed by every lane of the matrix
// for itself; V stays in the matrix's shared memory.
// Measured against a parallel Jacobi of the 12x12 by a warp (single-precision
// seed, double refinement), building included: 172 k barrier constraints 41.8
// -> 3.1 ms (FP64 issue), 98 k friction constraints 25.9 -> 1.4 ms, 338 barrier
// constraints (16 lanes each) 0.50 -> 0.17 ms (the chain of one matrix).

template <int W>
__device__ __forceinline__ void group_sync(unsigned mask)
{
    if (W > 1) __syncwarp(mask);
}

constexpr int kQRSteps = 30 * kRed;  // bound of the QR iteration (converges in about 1.7 per row)

// g: this lane's number in the matrix's group of W lanes, mask: the group's
template <int W>
static __device__ void psd_project(SMat H, int g, unsigned mask)
{
    double d[kRed], e[kRed];
    const double kSqrt2 = 1.4142135623730951;
    double keep[(kRed + W - 1) / W][kRed];  // the matrix as given
#pragma unroll
    for (int i = 0; i < (kRed + W - 1) / W; i++)
#pragma unroll
        for (int c = 0; c < kRed; c++)
            if (g + i * W < kRed && c <= g + i * W) keep[i][c] = H.full(g + i * W, c);
    group_sync<W>(mask);
    // (t_a - t_b) / sqrt 2 in the place of t_a
    for (int r = g; r < kRed; r += W)
        for (int c = 0; c < 3 && c <= r; c++) H.full(r, c) *= r < 3 ? 2.0 : kSqrt2;
    group_sync<W>(mask);
    // ---- tridiagonalisation: v_k in column k below the diagonal, its factor
    // beta_k on the diagonal, the update vector in row k above it
#pragma unroll 1
    for (int k = 0; k < kRed - 2; k++) {
        const double x1 = H.full(k + 1, k);
        double sg = 0;
        for (int i = k + 2; i < kRed; i++) sg = fma(H.full(i, k), H.full(i, k), sg);
        d[k] = H.full(k, k);
        group_sync<W>(mask);
        const double h = fma(x1, x1, sg);
        if (!(sg > 0.0) || h < 1e-290) {
            e[k] = x1;
            if (g == 0) H.full(k, k) = 0;
            group_sync<W>(mask);
            continue;
        }
        const double r = __dmul_rn(h, rsqrt(h));
        e[k] = x1 > 0 ? -r : r;
        const double v1 = x1 - e[k];
        const double beta = 1.0 / fma(fabs(x1), r, h);
        if (g == 0) {
            H.full(k + 1, k) = v1;
            H.full(k, k) = beta;
        }
        group_sync<W>(mask);
        // p = beta A v, then w = p - (beta / 2 v^T p) v
        for (int i = k + 1 + g; i < kRed; i += W) {
            double a = 0;
            for (int j = k + 1; j < kRed; j++) a = fma(i >= j ? H.full(i, j) : H.full(j, i), H.full(j, k), a);
            H.full(k, i) = beta * a;
        }
        group_sync<W>(mask);
        double vp = 0;
        for (int i = k + 1; i < kRed; i++) vp = fma(H.full(i, k), H.full(k, i), vp);
        group_sync<W>(mask);
        const double K = 0.5 * beta * vp;
        for (int i = k + 1 + g; i < kRed; i += W) H.full(k, i) = fma(-K, H.full(i, k), H.full(k, i));
        group_sync<W>(mask);
        for (int i = k + 1 + g; i < kRed; i += W) {
            const double vi = H.full(i, k), wi = H.full(k, i);
            for (int j = k + 1; j <= i; j++)
                H.full(i, j) = fma(-vi, H.full(k, j), fma(-wi, H.full(j, k), H.full(i, j)));
        }
        group_sync<W>(mask);
    }
    d[kRed - 2] = H.full(kRed - 2, kRed - 2);
    d[kRed - 1] = H.full(kRed - 1, kRed - 1);
    e[kRed - 2] = H.full(kRed - 1, kRed - 2);
    e[kRed - 1] = 0;
    group_sync<W>(mask);
    // ---- V = H_0 H_1 ... from the last reflection back, growing a row and
    // a column at a time; lanes take columns
    for (int r = kRed - 2 + g; r < kRed; r += W)
        for (int c = kRed - 2; c < kRed; c++) H.full(r, c) = r == c ? 1.0 : 0.0;
    group_sync<W>(mask);
#pragma unroll 1
    for (int k = kRed - 3; k >= 0; k--) {
        const double beta = H.full(k, k);
        for (int c = k + 1 + g; c < kRed; c += W) {
            double a = 0;
            for (int i = k + 1; i < kRed; i++) a = fma(H.full(i, k), H.full(i, c), a);
            a *= beta;
            for (int i = k + 1; i < kRed; i++) H.full(i, c) = fma(-a, H.full(i, k), H.full(i, c));
        }
        group_sync<W>(mask);
        // row and column k become the identity's
        for (int c = k + g; c < kRed; c += W) {
            H.full(k, c) = c == k ? 1.0 : 0.0;
            H.full(c, k) = c == k ? 1.0 : 0.0;
        }
        group_sync<W>(mask);
    }
    // ---- implicit QR on (d, e); an off-diagonal below rounding is set to
    // zero; lanes rotate their rows of V
    double norm = 0;
    for (int k = 0; k < kRed; k++) norm += fabs(d[k]) + fabs(e[k]);
    if (!(norm < INFINITY)) {
        for (int r = g; r < kRed; r += W)
            for (int c = 0; c <= r; c++) H.full(r, c) = norm - norm;  // NaN
        group_sync<W>(mask);
        return;
    }
    // scaled by a power of two to a norm of [1, 2): the shifts are single
    // precision; off-diagonals below 1e-17 of the norm are zero
    const long long ex = (__double_as_longlong(norm) >> 52) & 0x7ff;
    const bool scaled = ex > 0 && ex < 2046;
    const double scale = scaled ? __longlong_as_double((2046 - ex) << 52) : 1.0;
    const double unscale = scaled ? __longlong_as_double(ex << 52) : 1.0;
    for (int k = 0; k < kRed; k++) {
        d[k] *= scale;
        e[k] *= scale;
    }
    const double tiny = norm * scale * 1e-17;
    for (int k = 0; k + 1 < kRed; k++)
        if (fabs(e[k]) <= fma(1.1102230246251565e-16, fabs(d[k]) + fabs(d[k + 1]), tiny)) e[k] = 0;
#pragma unroll 1
    for (int step = 0; step < kQRSteps; step++) {
        int q = kRed - 1;
        while (q > 0 && (__double_as_longlong(e[q - 1]) << 1) == 0) q--;
        if (q == 0) break;
        int p = q - 1;
        while (p > 0 && (__double_as_longlong(e[p - 1]) << 1) != 0) p--;
        // the shift only steers the convergence: single precision
        const float eq = (float)e[q - 1], dl = 0.5f * (float)(d[q - 1] - d[q]);
        const float rt = sqrtf(fmaf(dl, dl, eq * eq));
        const float den = dl + (dl >= 0.0f ? rt : -rt);
        const double mu = d[q] - (double)(den != 0.0f ? __fdividef(eq, den) * eq : 0.0f);
        double x = d[p] - mu, z = e[p];
        double dk = d[p], ek = e[p];
#pragma unroll 1
        for (int k = p; k < q; k++) {
            // rotation of (k, k + 1) that takes (x, z) to (r, 0)
            const double h = fma(x, x, z * z);
            double c = 1, s = 0;
            if (h > 1e-290) {
                const double ir = rsqrt(h);
                c = x * ir;
                s = z * ir;
                if (k > p) {
                    const double r = h * ir;
                    e[k - 1] = fabs(r) <= fma(1.1102230246251565e-16, fabs(d[k - 1]) + fabs(dk), tiny) ? 0.0 : r;
                }
            } else if (k > p) {
                e[k - 1] = 0;
            }
            const double d1 = d[k + 1];
            const double t = __dmul_rn(fma(s, dk - d1, -2.0 * c * ek), s);  // dk - new dk
            const double cs = c * s, c2s2 = fma(c, c, -s * s);
            const double en = fma(cs, d1 - dk, c2s2 * ek);
            d[k] = dk - t;
            dk = d1 + t;
            d[k + 1] = dk;
            if (k + 1 < q) {
                z = s * e[k + 1];
                ek = c * e[k + 1];
                e[k + 1] = ek;
            }
            x = en;
            e[k] = en;
            for (int r = g; r < kRed; r += W) {
                const double a = H.full(r, k), b = H.full(r, k + 1);
                H.full(r, k) = fma(s, b, c * a);
                H.full(r, k + 1) = fma(c, b, -s * a);
            }
        }
        if (fabs(e[q - 1]) <= fma(1.1102230246251565e-16, fabs(d[q - 1]) + fabs(d[q]), tiny)) e[q - 1] = 0;
    }
    group_sync<W>(mask);
    // ---- the matrix minus its negative part, A + V max(-L, 0) V^T, lower
    // triangle: rounds relative to the negative part, and leaves a matrix
    // with no negative eigenvalue as it is
#pragma unroll
    for (int i = 0; i < (kRed + W - 1) / W; i++) {
        const int r = g + i * W;
        if (r >= kRed) break;
        double wz[kRed];
#pragma unroll
        for (int k = 0; k < kRed; k++) wz[k] = fmax(-d[k] * unscale, 0.0) * H.full(r, k);
#pragma unroll
        for (int c = 0; c < kRed; c++) {
            if (c > r) break;
            double a = 0;
#pragma unroll
            for (int k = 0; k < kRed; k++) a = fma(wz[k], H.full(c, k), a);
            keep[i][c] = fma(a, c >= 3 ? 1.0 : r < 3 ? 0.5 : 0.70710678118654757, keep[i][c]);
        }
    }
    group_sync<W>(mask);
#pragma unroll
    for (int i = 0; i < (kRed + W - 1) / W; i++) {
        const int r = g + i * W;
        if (r >= kRed) break;
#pragma unroll
        for (int c = 0; c < kRed; c++)
            if (c <= r) H.full(r, c) = keep[i][c];
    }
}

// reduced index and sign of a row of the full 12x12
__device__ __forceinline__ void full_row(int r, int& i, bool& neg)
{
    neg = r >= 6 && r < 9;
    i = r < 6 ? r : r < 9 ? r - 6 : r - 3;
}

// The warp writes the local Hessians of its `count` constraints from ci0 on
// (slots 0 .. count - 1 of base; bit s of built: slot s holds one), 144
// coalesced doubles each, to the full and the blocked output.
__device__ __forceinline__ void write_local_hessians(const double* base, int stride, unsigned built, int64_t ci0,
                                                     double* hess, double* blocks)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 0; o < 2; o++) {
        double* dst = o ? blocks : hess;
        if (!dst) continue;
        for (int k = lane; k < 144; k += 32) {
            const int r = o ? (k / 72) * 6 + (k % 36) / 6 : k / 12;
            const int c = o ? ((k / 36) & 1) * 6 + k % 6 : k % 12;
            int i, j;
            bool ni, nj;
            full_row(r, i, ni);
            full_row(c, j, nj);
            const double* src = base + (size_t)(max(i, j) * kRed + min(i, j)) * stride;
            for (unsigned b = built; b; b &= b - 1) {
                const int s = __ffs(b) - 1;
                const double v = src[s];
                dst[(ci0 + s) * 144 + k] = ni != nj ? -v : v;
            }
        }
    }
}

// One warp per block and per_warp constraints (a power of two) per warp: W =
// min(16, 32 / per_warp) lanes to each.  The lanes of a group build their
// constraint's terms (build(ci, H, g, group): true in the first when H holds a
// Hessian to project and write), the group projects it, the warp writes it.
template <int W, class Build>
__device__ __forceinline__ void local_terms(int64_t n, int per_warp, int flags, double* hess, double* blocks,
                                            double* smem, Build build)
{
    const int lane = threadIdx.x, slot = lane / W, g = lane % W;
    const int64_t ci0 = (int64_t)blockIdx.x * per_warp, ci = ci0 + slot;
    const int stride = per_warp | 1;
    SMat H { smem + slot, stride };
    const unsigned group = W == 32 ? 0xffffffffu : ((1u << (W & 31)) - 1u) << (slot * W);
    const bool built = slot < per_warp && ci < n && build(ci, H, g, group);
    if (!(flags & RIGC_HESS)) return;  // uniform over the block
    const unsigned leaders = __ballot_sync(0xffffffffu, built && g == 0);
    __syncwarp();
    if ((flags & RIGC_PROJECT_PSD) && ((leaders >> (slot * W)) & 1u)) psd_project<W>(H, g, group);
    __syncwarp();
    unsigned slots = 0;
#pragma unroll
    for (int s = 0; s < 32 / W; s++) slots |= ((leaders >> (s * W)) & 1u) << s;
    write_local_hessians(smem, stride, slots, ci0, hess, blocks);
}

// Generic deterministic assembly of per-constraint body-space terms: cgrad
// (n x 12, two 6-blocks per constraint) into grad (nb x 6) and cblocks
// (n x 4 x 36) into a block-sparse matrix (row_ptr, col, val).  nseg_dev
// points at two device ints: the gradient segment count and the number of
// Hessian blocks (read back by the caller after a sync).
int assemble_terms(Ctx& c, const int* bodies, int64_t n, const double* cgrad,
                   const double* cblocks, DevBuf& grad, DevBuf& row_ptr, DevBuf& col,
                   DevBuf& val, int32_t* nseg_dev, bool with_hess);

size_t local_terms_smem_bytes(int per_warp);
int local_terms_per_warp(int64_t n, int tuned);
int launch_body_frames(Ctx& c, const double* x);

} // namespace rigc

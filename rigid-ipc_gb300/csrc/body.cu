// Per-body inertial energy with its gradient and 6x6 Hessian.
//
// Replaces compute_energy_term / compute_body_energy with the default
// implicit Euler integration (src/problems/distance_barrier_rb_problem.cpp:
// 706-944): for a dynamic body with pose x = (q, theta), Q = R(theta),
//   E = 1/2 m q.q - m q.(q0 + h (v0 + h g))              (unless q is fixed)
//     + 1/2 tr(Q J Q^T) - tr(Q J (Q0 + h Qdot0)^T)        (unless theta is fixed)
// with J = diag(1/2 (-I0 + I1 + I2), ...) from the principal moments
// (compute_J, :253-259).  The rotational derivatives use dQ/dtheta and
// d2Q/dtheta2 from the closed-form body frame (rotation.cuh).  The position
// block of the Hessian is m I (already positive definite; the reference's
// project_to_psd at :767-768 leaves it unchanged).
#include <algorithm>

#include "common.cuh"
#include "rotation.cuh"
#include "sort.cuh"

namespace rigc {

// rot_rn by a warp: a half of the lanes for each sinc
__device__ __forceinline__ void warp_rot_rn(const double t[3], int lane, double R[9])
{
    const double f = lane < 16 ? 1.0 : 0.5;
    const double s = sinc_rn(norm3_rn(RMUL(t[0], f), RMUL(t[1], f), RMUL(t[2], f)));
    rot_from_sinc(t, __shfl_sync(0xffffffffu, s, 0), __shfl_sync(0xffffffffu, s, 16), R);
}

// A warp per body, or (many bodies) a thread.  Bound by one body's chain: some
// 2000 FP64 instructions by a thread, 43 us; by a warp (19 us) the two angles of both
// rotations, the frame's entries and the sums are dealt out to the lanes.
template <bool kWarp>
__global__ void __launch_bounds__(kWarp ? 32 : 128)
k_body_energy(const double* __restrict__ x, const int* __restrict__ type, int nb,
              rigc_body_state s, double g0, double g1, double g2, double h,
              double* __restrict__ energy, double* __restrict__ grad,
              double* __restrict__ hess)
{
    __shared__ double frame[kWarp ? kFrameDoubles : 1], sums[kWarp ? 10 : 1];
    const int b = kWarp ? blockIdx.x : blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const int lane = kWarp ? threadIdx.x : 0;
    constexpr int kStep = kWarp ? 32 : 1;
    double e = 0, g[6] = { 0, 0, 0, 0, 0, 0 }, H[7] = { 0, 0, 0, 0, 0, 0, 0 };  // m, the rotation's six
    if (type[b] == RIGC_BODY_DYNAMIC) {
        const int fixed = s.dof_fixed[b];
        const double m = s.mass[b];
        const double* q = x + 6 * b;
        const double* q0 = s.x_t0 + 6 * b;
        const double* v0 = s.v_t0 + 6 * b;
        const double grav[3] = { g0, g1, g2 };
        if ((fixed & 7) != 7) {
            double qq = 0, qh = 0;
            for (int i = 0; i < 3; i++) {
                double hat = q0[i] + h * (v0[i] + h * grav[i]);
                qq += q[i] * q[i];
                qh += q[i] * hat;
                g[i] = m * q[i] - m * hat;
            }
            H[0] = m;
            e += 0.5 * m * qq - m * qh;
        }
        if ((fixed & 56) != 56) {
            const double* I = s.moment + 3 * b;
            const double J[3] = { 0.5 * (-I[0] + I[1] + I[2]), 0.5 * (I[0] - I[1] + I[2]),
                                  0.5 * (I[0] + I[1] - I[2]) };
            const double t[3] = { q[3], q[4], q[5] }, t0[3] = { q0[3], q0[4], q0[5] };
            double Q0[9], own[kWarp ? 1 : kFrameDoubles], part[kWarp ? 1 : 10];
            double* F = kWarp ? frame : own;
            double* sum = kWarp ? sums : part;
            if (kWarp) {
                warp_body_frame(t, lane, F);
                warp_rot_rn(t0, lane, Q0);
                __syncwarp();
            } else {
                body_frame(t, F);
                rot_rn(t0, Q0);
            }
            const double* Qd = s.Qdot_t0 + 9 * b;
            // D = Q - T, T = Q0 + h Qdot0; E = sum_ik J_k (1/2 Q_ik^2 - Q_ik T_ik)
            double T[9], D[9];
            for (int k = 0; k < 9; k++) {
                T[k] = Q0[k] + h * Qd[k];
                D[k] = F[k] - T[k];
            }
            // the energy, three gradient entries, six of the Hessian
            for (int task = lane; task < 10; task += kStep) {
                double acc = 0;
                if (task == 0) {
                    for (int k = 0; k < 9; k++) acc += J[k % 3] * (0.5 * F[k] * F[k] - F[k] * T[k]);
                } else if (task < 4) {
                    const double* dA = F + 9 * task;
                    for (int k = 0; k < 9; k++) acc += J[k % 3] * dA[k] * D[k];
                } else {
                    const int p = task - 4, ia = p < 3 ? 0 : p < 5 ? 1 : 2, ic = p < 3 ? p : p < 5 ? p - 2 : 2;
                    const double *dA = F + 9 + 9 * ia, *dC = F + 9 + 9 * ic, *d2 = F + 36 + 9 * p;
                    for (int k = 0; k < 9; k++) acc += J[k % 3] * (d2[k] * D[k] + dA[k] * dC[k]);
                }
                sum[task] = acc;
            }
            if (kWarp) __syncwarp();
            e += sum[0];
            for (int k = 0; k < 3; k++) g[3 + k] = sum[1 + k];
            for (int k = 0; k < 6; k++) H[1 + k] = sum[4 + k];
        }
    }
    if (lane == 0) energy[b] = e;
    if (grad)
        for (int k = lane; k < 6; k += kStep) grad[6 * b + k] = g[k];
    if (hess)
        for (int k = lane; k < 36; k += kStep) {
            const int r = k / 6, c = k % 6;
            hess[36 * (size_t)b + k] = r < 3 || c < 3 ? (r == c ? H[0] : 0.0) : H[1 + sym_index(r - 3, c - 3)];
        }
}

// energy_host null: the energy is in c.h_scalars[8] after the stream's next wait
int body_energy(Ctx& c, const rigc_body_state& s, const double* x, const double gravity[3],
                double h, double* energy_host, double* grad, double* hess)
{
    const int nb = c.s.nb;
    cudaStream_t st = c.stream;
    RIGC_TRY(c.scratch[0].reserve((size_t)(nb + 1) * sizeof(double)));
    double* e = c.scratch[0].as<double>();
    RIGC_COUNT_LAUNCH();
    if (nb <= kWarpFrames)
        k_body_energy<true><<<(unsigned)std::max(nb, 1), 32, 0, st>>>(x, c.s.type, nb, s, gravity[0], gravity[1],
                                                                      gravity[2], h, e, grad, hess);
    else
        k_body_energy<false><<<grid_for(nb, 128), 128, 0, st>>>(x, c.s.type, nb, s, gravity[0], gravity[1],
                                                                gravity[2], h, e, grad, hess);
    RIGC_CUDA(cudaGetLastError());
    double* e_dev = reinterpret_cast<double*>(c.d_scalars.as<char>() + 2560);
    RIGC_TRY(sum_f64(e, nb, e_dev, c.scratch[1], st));
    RIGC_CUDA(cudaMemcpyAsync(c.h_scalars + 8, e_dev, sizeof(double), cudaMemcpyDeviceToHost, st));
    if (!energy_host) return RIGC_OK;
    RIGC_CUDA(cudaStreamSynchronize(st));
    *energy_host = c.h_scalars[8];
    return RIGC_OK;
}

} // namespace rigc

// gpt_adjoint.cu -- gradients of a loss of the SQP step with respect to the
// cost weights and the end-effector goal (the adjoint of the KKT solve).
//
// No reference counterpart (the reference has no derivatives of its solve).
// At an iterate xu the SQP step solves K(theta) [dz; lambda] = [g(theta); c]
// (the KKT system of gato_form_kkt / oldschur.cuh:966-1092) and proposes
// xu+ = xu - dz (the first line-search step, alpha_0 = -1, toplevel.cuh:409).
// For a loss l(xu+) with h = dl/d(dz) = -dl/dxu+, the adjoint solve
// K mu = [h; 0] (K is symmetric, so the same Schur complement and PCG serve)
// gives dl/dtheta = mu_z^T (dg/dtheta - dG/dtheta dz).  theta enters only the
// cost blocks of knot k through
//   v_k = q_ee J_k^T (p(q_k) - p*_k)            position-cost gradient (7)
//   Q_k = [v_k v_k^T, 0; 0, diag(qd)],  q_k = [v_k; qd .* qdot_k]
//   R_k = diag(r),  r_k = r .* u_k
// so with a = mu_q, d = dz_q the position part reduces to the adjoint of v_k,
//   w_k = a (1 - v_k^T d) - d (a^T v_k),
// and dl/dp*_k = -q_ee J_k w_k, dl/dq_ee = sum_k w_k^T J_k^T (p_k - p*_k),
// dl/dqd_i = sum_k mu_{k,7+i} (qdot_{k,i} - dz_{k,7+i}),
// dl/dr_i = sum_{k<N-1} mu_{k,u,i} (u_{k,i} - dz_{k,u,i}).
// The terminal block follows the forward model: with ref_terminal it is
// evaluated at x_{N-2} with target t = (a0^2, a0 a1, a0 a2), a = v_{N-2}
// (the reference kernel's overwritten goal), whose derivative flows back into
// v_{N-2}; otherwise at x_{N-1} with target p*_{N-1}.  Per-knot forward-kinematic
// quantities are recomputed, not stored.
#include "gpt_common.cuh"
#include "gpt_dyn.cuh"
#include "gpt_internal.h"

namespace gpt {

constexpr int ADJ_THREADS = 128;
constexpr int ADJ_PART = 16;  // per-knot partials: qd 0..6, r 7..13, q_ee 14

__device__ __forceinline__ void adj_v(const float *J, const float *p, const float *t, float qee, float *v)
{
#pragma unroll
    for (int i = 0; i < NQ; ++i)
        v[i] = qee * (J[3 * i] * (p[0] - t[0]) + J[3 * i + 1] * (p[1] - t[1]) + J[3 * i + 2] * (p[2] - t[2]));
}

// w = a (1 - v.d) - d (a.v): the adjoint of v in a^T v - a^T (v v^T) d
__device__ __forceinline__ void adj_w(const float *a, const float *d, const float *v, float *w)
{
    double vd = 0.0, av = 0.0;
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        vd += (double)v[i] * d[i];
        av += (double)a[i] * v[i];
    }
#pragma unroll
    for (int i = 0; i < NQ; ++i) w[i] = (float)((double)a[i] * (1.0 - vd) - (double)d[i] * av);
}

// One thread per knot (a warp per knot had one lane do the forward kinematics: 164 -> 16 us at 512 x 128).
__global__ void __launch_bounds__(ADJ_THREADS)
    adjoint_grad_kernel(BatchView bv, ProblemParams P, const float *__restrict__ xu, const float *__restrict__ goal,
                        const float *__restrict__ dz, const float *__restrict__ mu, float *__restrict__ grad_goal,
                        float *__restrict__ part)
{
    const int jend = bv.j0 + bv.total_knots;
    for (int j = bv.j0 + blockIdx.x * blockDim.x + threadIdx.x; j < jend; j += gridDim.x * blockDim.x) {
        const int b = bv.inst(j);
        if (!bv.active(b)) continue;
        const int N = bv.N(b), k = j - bv.off(b);
        if (k == N - 1) continue;  // the terminal knot is handled with knot N-2
        const bool terminal = (k == N - 2);
        const float *x0 = xu + (size_t)NX * j, *d0 = dz + (size_t)NX * j, *m0 = mu + (size_t)NX * j;
        const float *gl = goal + (size_t)6 * j;
        const float qee = P.q_ee;
        float q[NQ], mq[NQ], dq[NQ], p[3], Jac[3 * NQ], v[NQ], w[NQ], e[3];
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            q[i] = x0[i];
            mq[i] = m0[i];
            dq[i] = d0[i];
        }
        {
            JointTrig t;
            joint_trig(q, t);
            fk_lane<true>(t, p, Jac);
        }
#pragma unroll
        for (int dd = 0; dd < 3; ++dd) e[dd] = p[dd] - gl[dd];
        adj_v(Jac, p, gl, qee, v);
        adj_w(mq, dq, v, w);
        double gq = 0.0;                     // d l / d q_ee
        float gg_next[3] = {0.f, 0.f, 0.f};  // d l / d p*_{k+1} (terminal, spec mode)
        double qd_part[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) qd_part[i] = (double)m0[NQ + i] * ((double)x0[NQ + i] - (double)d0[NQ + i]);
        if (terminal) {
            // terminal cost block (knot N-1)
            const float *x1 = x0 + NX, *d1 = d0 + NX, *m1 = m0 + NX;
            const float *xt = P.ref_terminal ? x0 : x1;
            float tt[3], pt[3], Jt[3 * NQ], vt[NQ], wt[NQ], md[NQ], ddq[NQ];
            if (P.ref_terminal) {
                const float a0 = v[0];
                tt[0] = a0 * a0;
                tt[1] = a0 * v[1];
                tt[2] = a0 * v[2];
#pragma unroll
                for (int i = 0; i < 3; ++i) pt[i] = p[i];
#pragma unroll
                for (int i = 0; i < 3 * NQ; ++i) Jt[i] = Jac[i];
            } else {
                tt[0] = gl[6];
                tt[1] = gl[7];
                tt[2] = gl[8];
                float q1[NQ];
#pragma unroll
                for (int i = 0; i < NQ; ++i) q1[i] = x1[i];
                JointTrig t;
                joint_trig(q1, t);
                fk_lane<true>(t, pt, Jt);
            }
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                md[i] = m1[i];
                ddq[i] = d1[i];
            }
            adj_v(Jt, pt, tt, qee, vt);
            adj_w(md, ddq, vt, wt);
            // d l / d target = -q_ee J_t w_t
            float gt[3];
#pragma unroll
            for (int dd = 0; dd < 3; ++dd) {
                double a = 0.0;
#pragma unroll
                for (int i = 0; i < NQ; ++i) a += (double)Jt[3 * i + dd] * wt[i];
                gt[dd] = (float)(-(double)qee * a);
            }
            // direct q_ee dependence of v_t = q_ee J_t^T (p_t - t)
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                double a = 0.0;
#pragma unroll
                for (int dd = 0; dd < 3; ++dd) a += (double)Jt[3 * i + dd] * ((double)pt[dd] - (double)tt[dd]);
                gq += (double)wt[i] * a;
            }
            if (P.ref_terminal) {
                // t = (a0^2, a0 a1, a0 a2) with a = v_{N-2}: the target's adjoint flows into w_{N-2}
                w[0] += 2.f * v[0] * gt[0] + v[1] * gt[1] + v[2] * gt[2];
                w[1] += v[0] * gt[1];
                w[2] += v[0] * gt[2];
            } else {
#pragma unroll
                for (int dd = 0; dd < 3; ++dd) gg_next[dd] = gt[dd];
            }
            // terminal velocity cost qd .* qdot_t
#pragma unroll
            for (int i = 0; i < NQ; ++i)
                qd_part[i] += (double)m1[NQ + i] * ((double)xt[NQ + i] - (double)d1[NQ + i]);
        }
        // knot k: d l / d p*_k = -q_ee J_k w_k and the q_ee term w_k^T J_k^T e_k
        float *gk = grad_goal + (size_t)6 * j;
#pragma unroll
        for (int dd = 0; dd < 3; ++dd) {
            double a = 0.0;
#pragma unroll
            for (int i = 0; i < NQ; ++i) a += (double)Jac[3 * i + dd] * w[i];
            gk[dd] = (float)(-(double)qee * a);
            gk[3 + dd] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            double a = 0.0;
#pragma unroll
            for (int dd = 0; dd < 3; ++dd) a += (double)Jac[3 * i + dd] * e[dd];
            gq += (double)w[i] * a;
        }
        if (terminal) {
#pragma unroll
            for (int dd = 0; dd < 3; ++dd) {
                gk[6 + dd] = gg_next[dd];
                gk[9 + dd] = 0.f;
            }
        }
        float *pk = part + (size_t)ADJ_PART * j;
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            pk[i] = (float)qd_part[i];
            pk[NQ + i] = (float)((double)m0[NS + i] * ((double)x0[NS + i] - (double)d0[NS + i]));
        }
        pk[14] = (float)gq;
    }
}

// per instance: fixed-order FP64 sums of the per-knot partials (knots 0..N-2): thread (g, t) sums component t of the
// knots g, g + RED_GROUPS, ...; the groups' sums are added in order (wacc: added to wacc[15 b + t] instead).  One
// thread per component walked the horizon alone: 40 -> 6 us at 512 x 128, 30 -> 5 us for 33 instances of up to 96 knots.
constexpr int RED_GROUPS = 16;
__global__ void __launch_bounds__(ADJ_PART *RED_GROUPS)
    adjoint_reduce_kernel(BatchView bv, const float *__restrict__ part, float *__restrict__ grad_qd,
                          float *__restrict__ grad_r, float *__restrict__ grad_qee, float *__restrict__ wacc)
{
    __shared__ double sums[RED_GROUPS][ADJ_PART];
    const int b = bv.b0 + (int)blockIdx.x;
    if (!bv.active(b)) return;
    const int t = threadIdx.x % ADJ_PART, g = threadIdx.x / ADJ_PART;
    const int N = bv.N(b), kb = bv.off(b);
    double a = 0.0;
    if (t < 15)
        for (int k = g; k < N - 1; k += RED_GROUPS) a += (double)part[(size_t)ADJ_PART * (kb + k) + t];
    sums[g][t] = a;
    __syncthreads();
    if (g > 0 || t >= 15) return;
    for (int i = 1; i < RED_GROUPS; ++i) a += sums[i][t];
    if (wacc) wacc[(size_t)15 * b + t] += (float)a;
    else if (t < NQ) grad_qd[(size_t)NQ * b + t] = (float)a;
    else if (t < NQ + NC) grad_r[(size_t)NC * b + t - NQ] = (float)a;
    else grad_qee[b] = (float)a;
}

// out = a + alpha * x (a == nullptr: out = alpha * x)
__global__ void axpy_kernel(int n, float alpha, const float *__restrict__ x, const float *__restrict__ a,
                            float *__restrict__ out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = a ? fmaf(alpha, x[i], a[i]) : alpha * x[i];
}

cudaError_t launch_adjoint_grad(const BatchView &bv, const ProblemParams &P, const float *xu, const float *goal,
                                const float *dz, const float *mu, float *grad_goal, float *part, float *grad_qd,
                                float *grad_r, float *grad_qee, int num_sms, cudaStream_t s, float *wacc)
{
    if (bv.total_knots <= 0) return cudaSuccess;
    // few knots: a warp per block, so that they spread over the SMs
    const int threads = bv.total_knots < num_sms * ADJ_THREADS ? 32 : ADJ_THREADS;
    int blocks = (bv.total_knots + threads - 1) / threads;
    if (blocks > num_sms * 16) blocks = num_sms * 16;
    adjoint_grad_kernel<<<blocks, threads, 0, s>>>(bv, P, xu, goal, dz, mu, grad_goal, part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    adjoint_reduce_kernel<<<bv.B, ADJ_PART * RED_GROUPS, 0, s>>>(bv, part, grad_qd, grad_r, grad_qee, wacc);
    return cudaGetLastError();
}

cudaError_t launch_axpy(int n, float alpha, const float *x, const float *a, float *out, int num_sms, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    int blocks = (n + 255) / 256;
    if (blocks > num_sms * 8) blocks = num_sms * 8;
    axpy_kernel<<<blocks, 256, 0, s>>>(n, alpha, x, a, out);
    return cudaGetLastError();
}

size_t adjoint_part_floats() { return ADJ_PART; }

}  // namespace gpt

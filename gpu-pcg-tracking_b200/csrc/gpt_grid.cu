// gpt_grid.cu -- batched rigid-body library kernels of the iiwa14 (the standalone GRiD kernels the
// reference ships, rbdfiles/iiwa_eepos_grid.cuh, called one state per launch there):
//
//   ee_pose_kernel  end_effector_positions_kernel (:2091-2110, inner :2015-2090): xyz + roll /
//                   pitch / yaw per row, one thread per row (generateeepos.cu:101-107 launches it
//                   once per trajectory row)
//   fd_kernel       forward_dynamics (:4351-4395): qdd = M^{-1}(u - c(q, qd)), gravity 0, one group
//                   of 8 lanes per row (fd_group); fd_lane_kernel one lane per row
//   fd_grad_kernel  forwardDynamicsAndGradient (rbdfiles/iiwa_eepos_plant.cuh:130-160): qdd and
//                   df/du = [-M^{-1} dID/dq, -M^{-1} dID/dqd, M^{-1}] (7 x 21, column-major), one
//                   half-warp per row with the lane roles of kkt_kernel; fd_grad_lane_kernel one lane per row
//
// Rows are read with a caller-given stride, so the rows of a trajectory (21 floats: x, u) and plain
// states (14 floats) are both accepted.
#include "gpt_common.cuh"
#include "gpt_dyn.cuh"
#include "gpt_fdlane.cuh"
#include "gpt_internal.h"

namespace gpt {

__global__ void __launch_bounds__(128) ee_pose_kernel(uint32_t n, const float *__restrict__ x, uint32_t stride,
                                                      float *__restrict__ pose)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float q[NQ];
#pragma unroll
    for (int j = 0; j < NQ; ++j) q[j] = x[(size_t)stride * i + j];
    JointTrig t;
    joint_trig(q, t);
    float p[6];
    fk_pose_lane(t, p);
#pragma unroll
    for (int j = 0; j < 6; ++j) pose[(size_t)6 * i + j] = p[j];
}

__global__ void __launch_bounds__(128) fd_kernel(uint32_t n, const float *__restrict__ xu, uint32_t stride,
                                                 float *__restrict__ qdd)
{
    const int lane = threadIdx.x & 31, m = lane & 7, base = lane & ~7;
    const uint32_t raw = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const bool live = raw < n;
    const uint32_t i = live ? raw : 0u;  // groups past the end follow row 0 (all lanes shuffle) and store nothing
    float q[NQ], qd[NQ], u[NC];
    const float *r = xu + (size_t)stride * i;
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
        q[j] = r[j];
        qd[j] = r[NQ + j];
        u[j] = r[NS + j];
    }
    double col[NQ];
    fd_group(q, qd, u, col, m, base);
    if (live && m == 7) {
#pragma unroll
        for (int j = 0; j < NQ; ++j) qdd[(size_t)NQ * i + j] = (float)col[j];
    }
}

struct FdgSmem {
    float x[NS], u[NC];
    JointTrig trig;
    float M[CC], cb[NQ], Minv[CC], qdd[NQ], dc[NQ * NS];
};
constexpr int FDG_WARPS = 4;

__global__ void __launch_bounds__(32 * FDG_WARPS)
    fd_grad_kernel(uint32_t n, const float *__restrict__ xu, uint32_t stride, float *__restrict__ qdd_out,
                   float *__restrict__ df_out)
{
    __shared__ FdgSmem sm_all[2 * FDG_WARPS];
    const int lane = threadIdx.x & 31, half = lane >> 4, hl = lane & 15;
    FdgSmem &sm = sm_all[2 * (threadIdx.x >> 5) + half];
    const uint32_t raw = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const bool live = raw < n;
    const uint32_t row = live ? raw : 0u;  // half-warps past the end follow row 0 and store nothing
    for (int i = hl; i < NX; i += 16) {
        const float v = xu[(size_t)stride * row + i];
        if (i < NS) sm.x[i] = v;
        else sm.u[i - NS] = v;
    }
    __syncwarp();
    if (hl < NQ) sincosf(sm.x[hl], &sm.trig.s[hl], &sm.trig.c[hl]);
    __syncwarp();
    const JointTrig trig = sm.trig;
    {  // mass-matrix columns (lanes 0..6), bias force (lane 7)
        float qd[NQ], qdd[NQ], tau[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            qd[i] = (hl == 7) ? sm.x[NQ + i] : 0.f;
            qdd[i] = (hl == i) ? 1.f : 0.f;
        }
        rnea<false>(trig, qd, qdd, -1, -1, tau, nullptr);
        if (hl < NQ) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) sm.M[NQ * hl + r] = tau[r];
        } else if (hl == NQ) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) sm.cb[r] = tau[r];
        }
    }
    __syncwarp();
    {  // Minv (lanes 7..13), qdd (lane 14): FP64 Gauss-Jordan on [M | I | u - c]
        double col[NQ];
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            double v = 0.0;
            if (hl < NQ) v = 0.5 * ((double)sm.M[NQ * hl + r] + (double)sm.M[NQ * r + hl]);
            else if (hl < 2 * NQ) v = (r == hl - NQ) ? 1.0 : 0.0;
            else if (hl == 2 * NQ) v = (double)sm.u[r] - (double)sm.cb[r];
            col[r] = v;
        }
        gj7_group(col, 16 * half);
        if (hl >= NQ && hl < 2 * NQ) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) sm.Minv[NQ * (hl - NQ) + r] = (float)col[r];
        } else if (hl == 2 * NQ) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) sm.qdd[r] = (float)col[r];
        }
    }
    __syncwarp();
    {  // dID/dq_j (lanes 0..6), dID/dqd_j (lanes 7..13) at (q, qd, qdd)
        float qd[NQ], qdd[NQ], tau[NQ], dtau[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            qd[i] = sm.x[NQ + i];
            qdd[i] = sm.qdd[i];
        }
        const int dq_dir = (hl < NQ) ? hl : -1;
        const int dqd_dir = (hl >= NQ && hl < NS) ? hl - NQ : -1;
        rnea<true>(trig, qd, qdd, dq_dir, dqd_dir, tau, dtau);
        if (hl < NS) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) sm.dc[NQ * hl + r] = dtau[r];
        }
    }
    __syncwarp();
    if (!live) return;
    if (hl < NQ) qdd_out[(size_t)NQ * row + hl] = sm.qdd[hl];
    for (int e = hl; e < NQ * NX; e += 16) {
        float v;
        if (e < NQ * NS) {
            const int col = e / NQ, r = e - NQ * col;
            float acc = 0.f;
#pragma unroll
            for (int t = 0; t < NQ; ++t) acc += sm.Minv[r + NQ * t] * sm.dc[NQ * col + t];
            v = -acc;
        } else {
            v = sm.Minv[e - NQ * NS];
        }
        df_out[(size_t)NQ * NX * row + e] = v;
    }
}

// The same with one row per lane (gpt_fdlane.cuh), eight warps per SM (255 registers a thread, 26 KB of shared memory a
// warp).  200,003 rows: 128 us against the half-warp form's 437, both cut by the issue of the tangent passes and their
// latency (the rows' 685 bytes would take 21 us); two warps per CTA fill the last wave best (four 1%
// more, eight 11%).
constexpr int FDGL_WARPS = 2;

__global__ void __launch_bounds__(32 * FDGL_WARPS, 8 / FDGL_WARPS)
    fd_grad_lane_kernel(uint32_t n, const float *__restrict__ xu, uint32_t stride, float *__restrict__ qdd_out,
                        float *__restrict__ df_out)
{
    extern __shared__ float4 fdgl_dyn_smem[];
    const int lane = threadIdx.x & 31;
    FdLaneSmem &sm = reinterpret_cast<FdLaneSmem *>(fdgl_dyn_smem)[threadIdx.x >> 5];
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31);
    const bool valid = i0 + lane < n;  // lanes past the end follow the last row and store nothing
    const uint32_t mask = __ballot_sync(0xffffffffu, valid);
    const float *x = xu + (size_t)stride * (valid ? i0 + lane : n - 1);
    float q[NQ], qd[NQ], u[NC], qdd[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        q[i] = x[i];
        qd[i] = x[NQ + i];
        u[i] = x[NS + i];
    }
    JointTrig t;
    joint_trig(q, t);
    fd_gradient_lane(t, qd, u, qdd, sm, lane, [&](auto blk, int col, const float (&v)[NQ]) {
        store_rows<NQ, NQ * NX>(sm.out, v, df_out + NQ * NX * i0 + CC * blk.block + NQ * col, mask, lane);
    });
    store_rows<NQ, NQ>(sm.out, qdd, qdd_out + NQ * i0, mask, lane);
}

cudaError_t launch_fd_grad(uint32_t n, const float *xu, uint32_t stride, float *qdd, float *df, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    // One row per lane from FDGL_MIN rows on: up to four warps per SM (18,944 rows) that form takes 19.5 us whatever the
    // number of rows, the half-warp form 2.5 us per 1,000 rows beyond its own 4 (8,000 rows 23.6 against 19.4 us, 16,000
    // rows 40.3 against 19.5)
    constexpr uint32_t FDGL_MIN = 8192;
    if (n >= FDGL_MIN) {
        constexpr int per = 32 * FDGL_WARPS;
        const size_t smem = sizeof(FdLaneSmem) * FDGL_WARPS;
        const cudaError_t e = ensure_func_attrs((const void *)fd_grad_lane_kernel, smem);
        if (e != cudaSuccess) return e;
        fd_grad_lane_kernel<<<(unsigned)(((size_t)n + per - 1) / per), per, smem, s>>>(n, xu, stride, qdd, df);
        return cudaGetLastError();
    }
    fd_grad_kernel<<<(unsigned)(((size_t)n * 16 + 32 * FDG_WARPS - 1) / (32 * FDG_WARPS)), 32 * FDG_WARPS, 0, s>>>(
        n, xu, stride, qdd, df);
    return cudaGetLastError();
}

cudaError_t launch_ee_pose(uint32_t n, const float *x, uint32_t stride, float *pose, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    ee_pose_kernel<<<(n + 127) / 128, 128, 0, s>>>(n, x, stride, pose);
    return cudaGetLastError();
}

// Forward dynamics with one row per lane (gpt_fdlane.cuh): the mass matrix two columns at a time in packed FP32, the FP64
// solve in registers.  200,003 rows: 24.6 us against 78 with eight lanes per row, one of which each evaluates a column
// (the rows' 112 bytes take 3.5 us; bound by issue).
constexpr int FDL_WARPS = 4;

__global__ void __launch_bounds__(32 * FDL_WARPS, 4)
    fd_lane_kernel(uint32_t n, const float *__restrict__ xu, uint32_t stride, float *__restrict__ qdd_out)
{
    __shared__ struct {
        float M[CC][32], out[NS * 34];
    } sm_all[FDL_WARPS];
    auto &sm = sm_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31);
    const bool valid = i0 + lane < n;  // lanes past the end follow the last row and store nothing
    const uint32_t mask = __ballot_sync(0xffffffffu, valid);
    const float *x = xu + (size_t)stride * (valid ? i0 + lane : n - 1);
    float q[NQ], qd[NQ], u[NC], qdd[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        q[i] = x[i];
        qd[i] = x[NQ + i];
        u[i] = x[NS + i];
    }
    JointTrig t;
    joint_trig(q, t);
    fd_lane(t, qd, u, qdd, sm.M, lane);
    store_rows<NQ, NQ>(sm.out, qdd, qdd_out + NQ * i0, mask, lane);
}

cudaError_t launch_fd(uint32_t n, const float *xu, uint32_t stride, float *qdd, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    // up to 37,888 rows (four CTAs per SM) the lane form takes 8 us, launch included, the eight-lane form 8.4 at 4095 rows
    // and 0.4 us more per 1,000
    constexpr uint32_t FDL_MIN = 4096;
    if (n >= FDL_MIN) {
        constexpr int per = 32 * FDL_WARPS;
        fd_lane_kernel<<<(unsigned)(((size_t)n + per - 1) / per), per, 0, s>>>(n, xu, stride, qdd);
        return cudaGetLastError();
    }
    fd_kernel<<<(unsigned)(((size_t)n * 8 + 127) / 128), 128, 0, s>>>(n, xu, stride, qdd);
    return cudaGetLastError();
}

}  // namespace gpt

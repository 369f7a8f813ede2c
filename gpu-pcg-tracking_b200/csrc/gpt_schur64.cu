// gpt_schur64.cu -- the SQP loop's and the adjoints' Schur complement in FP64 (packed rows for the exact-
// preconditioner PCG), and its right-hand side alone for another gradient on the same system.
//
// The block row of gpt_schur.cu with every product, gamma and the stored row in FP64 (PK64 doubles per knot: left
// block 196 column-major, lower triangle of the diagonal block 105, pad).  FP32 formation perturbs S by ~10 eps32
// relative per entry, which cond(S) ~1e7 turns into ~1e-2 relative error of the solution; FP64 formation leaves
// only the FP32 rounding of the KKT data (C, g, c).
//
// Input: kkt_kernel's C, g, c.  Its cost blocks are functions of these: Q_k = [v v^T, 0; 0, QD I] with
// v = g_k[0..6] (each product rounded to FP32, as kkt_kernel writes it to G) and R_k = R_COST I, so G is not read.
//
// One warp per run of rows.  The 7x7 position inverses (v v^T + rho I)^{-1} of four knots are formed at once, one
// per group of eight lanes (lane m < 7 holds column m), by in-place Gauss-Jordan with 2x2 block pivots: the
// chain of four dependent steps, not its arithmetic, is what an inverse costs (measured alone, one per
// warp: 4.4 k cycles).  A row is then
//   theta = X diag(Qt_{k-1}^{-1}, Rt_{k-1}^{-1}) X^T + Qt_k^{-1},  X = [-A_{k-1}, -B_{k-1}] (14 x 21, as C stores it)
// on the FP64 tensor cores (K padded to 24): the position columns of phi = (-A) Qt^{-1} are a product (4 mma),
// the velocity and control columns a scaling; theta's three tiles (symmetric) take 18 mma, and row 14 of the
// padded X^T is [q; r]_{k-1}, so that column 14 of the product is gamma's sum.  Every operand is read from shared
// memory once, as FP32.
#include "gpt_common.cuh"
#include "gpt_internal.h"

namespace gpt {

// Pivot test: (Q + rho I) and (R + rho I) must be positive definite, so every pivot must be positive and not vanish
// against the diagonal entry it came from (a relative 1e-13 catches a singular matrix whose exact zero pivot
// rounding turned into a tiny number of either sign; NaN fails too)
constexpr double PIVOT_REL_MIN = 1e-13;

// In-place inverse of the 7x7 SPD matrix of each group of eight lanes: lane m < 7 of the group holds column m (lane 7
// takes the shuffles only).  2x2 block pivots {0,1}, {2,3}, {4,5} and the scalar pivot 6; diag: the lane's
// own diagonal entry.  Returns whether every pivot passed the test (the same on the group's lanes).
__device__ __forceinline__ bool group_inverse7(double (&a)[NQ], double diag, int m, int base)
{
    bool ok = true;
#pragma unroll
    for (int p = 0; p + 1 < NQ; p += 2) {
        double u0[NQ], u1[NQ];  // columns p, p + 1
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            u0[r] = __shfl_sync(0xffffffffu, a[r], base + p);
            u1[r] = __shfl_sync(0xffffffffu, a[r], base + p + 1);
        }
        const double d0 = __shfl_sync(0xffffffffu, diag, base + p), d1 = __shfl_sync(0xffffffffu, diag, base + p + 1);
        const double x = u0[p], y = u0[p + 1], z = u1[p + 1], det = fma(x, z, -y * y);
        ok = ok && (d0 > 0.0) && (d1 > 0.0) && (x > PIVOT_REL_MIN * d0) && (det > PIVOT_REL_MIN * d1 * x);
        const double rd = rcp_newton(det), i00 = z * rd, i01 = -y * rd, i11 = x * rd;
        const bool c0 = m == p, c1 = m == p + 1, piv = c0 || c1;
        const double w0 = piv ? (c0 ? 1.0 : 0.0) : a[p], w1 = piv ? (c1 ? 1.0 : 0.0) : a[p + 1];
        const double n0 = fma(i00, w0, i01 * w1), n1 = fma(i01, w0, i11 * w1);
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            a[r] = r == p ? n0 : (r == p + 1 ? n1 : fma(-u0[r], n0, fma(-u1[r], n1, piv ? 0.0 : a[r])));
    }
    constexpr int p = NQ - 1;
    double u[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) u[r] = __shfl_sync(0xffffffffu, a[r], base + p);
    const double d0 = __shfl_sync(0xffffffffu, diag, base + p);
    ok = ok && (d0 > 0.0) && (u[p] > PIVOT_REL_MIN * d0);
    const double rd = rcp_newton(u[p]);
    const bool piv = m == p;
    const double n0 = piv ? rd : a[p] * rd;
#pragma unroll
    for (int r = 0; r < p; ++r) a[r] = fma(-u[r], n0, piv ? 0.0 : a[r]);
    a[p] = n0;
    return ok;
}

constexpr int S64_WARPS = 4;
// a row's staged inputs (floats): C_{k-1} (14 x 21), [q; r]_{k-1}, q_k, c_k
constexpr int SI_G = C_STRIDE, SI_Q = SI_G + NX, SI_C = SI_Q + NS, SI_N = SI_C + NS + 1;
struct Schur64Warp {
    double inv[8][GC64];  // compact inverses (gpt_common.cuh) of knot j at [j & 7]
    float in[2][SI_N];
};
static_assert(SI_N % 2 == 0, "8-byte copies of C");

__device__ __forceinline__ void cp_async8(void *sdst, const void *gsrc)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(sdst)), "l"(gsrc)
                 : "memory");
}

__global__ void __launch_bounds__(32 * S64_WARPS, 5)
    schur64_kernel(BatchView bv, float qd_cost, float r_cost, const float *__restrict__ Cm,
                   const float *__restrict__ g, const float *__restrict__ c, double *__restrict__ S64,
                   double *__restrict__ gamma64, double *__restrict__ Ginv64c)
{
    __shared__ __align__(16) Schur64Warp smem_all[S64_WARPS];
    const int lane = threadIdx.x & 31;
    Schur64Warp &sm = smem_all[threadIdx.x >> 5];
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    // a contiguous run of rows per warp, so that a knot's inverse serves its own row and the next one
    const int chunk = (bv.total_knots + nw - 1) / nw;
    const int jbeg = bv.j0 + gw * chunk, jend = min(jbeg + chunk, bv.j0 + bv.total_knots);
    if (jbeg >= jend) return;

    // row j's inputs into sm.in[buf]; opens: the first row of an instance, which has no C
    auto stage = [&](int j, int buf, bool opens) {
        if (j < jend) {
            float *in = sm.in[buf];
            if (!opens) {
                const float *src = Cm + (size_t)C_STRIDE * (j - 1);
#pragma unroll
                for (int i = 0; i < C_STRIDE / 2; i += 32)
                    if (i + lane < C_STRIDE / 2) cp_async8(in + 2 * (i + lane), src + 2 * (i + lane));
                if (lane < NX) cp_async4(in + SI_G + lane, g + (size_t)NX * (j - 1) + lane);
            }
            if (lane < NS) {
                cp_async4(in + SI_Q + lane, g + (size_t)NX * j + lane);
                cp_async4(in + SI_C + lane, c + (size_t)NS * j + lane);
            }
        }
        cp_async_commit();
    };
    // the compact inverses of knots jb .. jb + 3 (those below jend), one per eight lanes
    auto invert = [&](int jb) {
        const int m = lane & 7, base = lane & ~7, mine = jb + (lane >> 3), j = min(mine, jend - 1);
        const int b = bv.inst(j);
        const double rho = (double)bv.st[b].rho;
        const bool last = j - bv.off(b) == bv.N(b) - 1;
        const float *v = g + (size_t)NX * j;
        float vf[NQ];
#pragma unroll
        for (int r = 0; r < NQ; ++r) vf[r] = v[r];
        const float vm = v[m < NQ ? m : 0];
        double a[NQ], diag = 0.0;
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            a[r] = (double)__fmul_rn(vf[r], vm) + (r == m ? rho : 0.0);
            if (r == m) diag = a[r];
        }
        const double dv = (double)qd_cost + rho, dc = (double)r_cost + rho;
        bool ok = group_inverse7(a, diag, m, base);
        ok = ok && dv > 0.0 && (last || dc > 0.0);
        const double rv = rcp_newton(dv), rc = last ? 0.0 : rcp_newton(dc);
        __syncwarp();
        if (mine < jend) {
            double *o = sm.inv[mine & 7];
            if (m < NQ) {
#pragma unroll
                for (int r = 0; r < NQ; ++r) o[GC_POS + NQ * m + r] = a[r];
                o[GC_VEL + m] = rv;
                o[GC_CTL + m] = rc;
            } else {
                o[0] = 0.0;
                if (!ok && bv.active(b)) atomicOr(&bv.st[b].exit_flags, GPT_EXIT_FACTOR);
            }
        }
        __syncwarp();
    };

    const int lg = lane >> 2, lt = lane & 3;
    // the instance of the current row: its first knot, the knot after its last, whether it runs
    int b = bv.inst(jbeg), b0 = bv.off(b), b1 = b0 + bv.N(b);
    bool act = bv.active(b);
    stage(jbeg, 0, jbeg == b0);
    int have = jbeg > b0 ? jbeg - 2 : jbeg - 1;  // inverses are formed up to this knot (row jbeg needs its predecessor's)
    for (int j = jbeg; j < jend; ++j) {
        const int buf = (j - jbeg) & 1;
        if (j == b1) {
            b = bv.inst(j);
            b0 = j;
            b1 = b0 + bv.N(b);
            act = bv.active(b);
        }
        stage(j + 1, buf ^ 1, j + 1 == b1);
        if (have < j) {
            invert(have + 1);
            have += 4;
        }
        cp_async_wait<1>();
        __syncwarp();
        if (act) {
            const int k = j - b0;
            const float *in = sm.in[buf];
            const double *io = sm.inv[j & 7], *ip = sm.inv[(j - 1) & 7];
            double *Pk = S64 + (size_t)PK64 * j;
            double *Lk = Pk, *Dk = Pk + SS;
            double th[3][2] = {};  // tiles (0,0), (0,1), (1,1) of theta without Qt_k^{-1}, column 14 gamma's sum
            if (k > 0) {
                // X fragments: x[I][kk] = X(8 I + g, 4 kk + t); row 14 is [q; r]_{k-1}
                const float *p0 = in + lg, *p1 = lg < 6 ? in + 8 + lg : in + SI_G;
                const int s1 = lg < 6 ? NS : 1;
                double x[2][6];
#pragma unroll
                for (int kk = 0; kk < 6; ++kk) {
                    const int K = kk < 5 ? 4 * kk + lt : 20;
                    const bool in_k = kk < 5 || lt == 0;
                    const float f0 = p0[NS * K], f1 = p1[s1 * K];
                    x[0][kk] = in_k ? (double)f0 : 0.0;
                    x[1][kk] = in_k && lg < 7 ? (double)f1 : 0.0;
                }
                // phi's columns 0 .. 7: the position inverse and the first velocity entry
                double ph[2][2] = {};
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) {
                    const int K = 4 * kk + lt;
                    const double pv = ip[GC_POS + (K < NQ ? K : 0) + NQ * (lg < NQ ? lg : 0)], dv = ip[GC_VEL];
                    const double bq = K < NQ && lg < NQ ? pv : (K == NQ && lg == NQ ? dv : 0.0);
                    mma884_f64(ph[0], x[0][kk], bq);
                    mma884_f64(ph[1], x[1][kk], bq);
                }
#pragma unroll
                for (int I = 0; I < 2; ++I)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (I == 0 || lg < 6) Lk[8 * I + lg + NS * (2 * lt + e)] = -ph[I][e];
                // the other columns of phi and (-B) Rt^{-1}: scalings (the store of phi's below)
#pragma unroll
                for (int kk = 0; kk < 6; ++kk) {
                    double y[2];
                    if (kk < 2) {  // accumulator layout -> operand layout, within the quad
                        const int src = (lane & ~3) | (2 * kk + (lt >> 1));
#pragma unroll
                        for (int I = 0; I < 2; ++I) {
                            const double q0 = __shfl_sync(0xffffffffu, ph[I][0], src);
                            const double q1 = __shfl_sync(0xffffffffu, ph[I][1], src);
                            y[I] = (lt & 1) ? q1 : q0;
                        }
                    } else {
                        const int K = kk < 5 ? 4 * kk + lt : 20;
                        const double sc = ip[GC_VEL - NQ + K];  // velocity, then control diagonal
                        y[0] = x[0][kk] * sc;
                        y[1] = x[1][kk] * sc;
                    }
                    mma884_f64(th[0], y[0], x[0][kk]);
                    mma884_f64(th[1], y[0], x[1][kk]);
                    mma884_f64(th[2], y[1], x[1][kk]);
                }
                const double dv = ip[GC_VEL];
#pragma unroll
                for (int i = 0; i < 6 * NS; i += 32)
                    if (i + lane < 6 * NS) Lk[8 * NS + i + lane] = -((double)in[8 * NS + i + lane] * dv);
            } else {
                for (int e = lane; e < SS; e += 32) Lk[e] = 0.0;  // no left block in row 0
            }
            // the diagonal block's lower triangle, -(theta + Qt_k^{-1}): element (i, jj) of the tiles
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = lg, jj = 2 * lt + e, i1 = 8 + lg, j1 = 8 + jj;
                const double pv = io[GC_POS + (i < NQ ? i : 0) + NQ * (jj < NQ ? jj : 0)], dv = io[GC_VEL];
                if (jj <= i)
                    Dk[((i * (i + 1)) >> 1) + jj] = -(th[0][e] + (i < NQ ? pv : (jj == NQ ? dv : 0.0)));
                if (j1 < NS) {
                    Dk[((j1 * (j1 + 1)) >> 1) + i] = -th[1][e];
                    if (i1 < NS && j1 <= i1) Dk[((i1 * (i1 + 1)) >> 1) + j1] = -(th[2][e] + (i1 == j1 ? dv : 0.0));
                }
            }
            // gamma = -(Qt_k^{-1} q_k - c_k + theta's column 14), rows g and 8 + g on the lanes t = 3
            if (lt == 3) {
                const float *q = in + SI_Q, *cc = in + SI_C;
                double s = 0.0;
                if (lg < NQ) {
#pragma unroll
                    for (int r = 0; r < NQ; ++r) s = fma(io[GC_POS + lg + NQ * r], (double)q[r], s);
                } else {
                    s = io[GC_VEL] * (double)q[NQ];
                }
                const double c0 = k > 0 ? (double)cc[lg] : 0.0;
                gamma64[(size_t)NS * j + lg] = -((s - c0) + th[1][0]);
                if (lg < 6) {
                    const double c1 = k > 0 ? (double)cc[8 + lg] : 0.0;
                    gamma64[(size_t)NS * j + 8 + lg] = -((io[GC_VEL] * (double)q[8 + lg] - c1) + th[2][0]);
                }
            }
            if (lane == 0) Pk[PK64 - 1] = 0.0;
            // the knot's inverses for dz
            double *dc = Ginv64c + (size_t)GC64 * j;
            dc[lane] = io[lane];
            dc[lane + 32] = io[lane + 32];
        }
        __syncwarp();  // sm.in[buf] and the inverses have been read
    }
    cp_async_wait<0>();
}

// gamma of the rows in S64 for another gradient g and defect c (null: 0): gamma_k = -(Qt_k^{-1} q_k - c_k + phi_k q_{k-1} +
// (-B) Rt^{-1} r_{k-1}), phi_k = -(left block).  One warp per knot: lane pair (i, h) takes row i, half h of the columns.
__global__ void __launch_bounds__(128)
    schur64_gamma_kernel(BatchView bv, const double *__restrict__ S64, const double *__restrict__ Ginv64c,
                         const float *__restrict__ Cm, const float *__restrict__ g, const float *__restrict__ c,
                         double *__restrict__ gamma64)
{
    const int lane = threadIdx.x & 31, i = lane >> 1 < NS ? lane >> 1 : NS - 1, h = lane & 1;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int j = bv.j0 + gw; j < bv.j0 + bv.total_knots; j += nw) {
        const int b = bv.inst(j);
        if (!bv.active(b)) continue;
        const bool first = j == bv.off(b);
        const double *io = Ginv64c + (size_t)GC64 * j;
        const float *q = g + (size_t)NX * j;
        // the halves' sums: h = 0 the position inverse's row and phi's even columns, h = 1 the rest
        double s = 0.0;
        if (i >= NQ) s = h ? io[GC_VEL + i - NQ] * (double)q[i] : 0.0;
        else if (h == 0)
#pragma unroll
            for (int r = 0; r < NQ; ++r) s = fma(io[GC_POS + i + NQ * r], (double)q[r], s);
        if (h && c && !first) s -= (double)c[(size_t)NS * j + i];
        if (!first) {
            const double *L = S64 + (size_t)PK64 * j + i, *ip = io - GC64;
            const float *qp = q - NX, *B = Cm + (size_t)C_STRIDE * (j - 1) + SS + i;
#pragma unroll
            for (int r = 0; r < NQ; ++r) {
                const int col = 2 * r + h;
                s = fma(-L[NS * col], (double)qp[col], s);
            }
#pragma unroll
            for (int r = 0; r < NC; ++r)
                if ((r & 1) == h) s = fma((double)B[NS * r] * ip[GC_CTL + r], (double)qp[NS + r], s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (h == 0 && lane < 2 * NS) gamma64[(size_t)NS * j + i] = -s;
    }
}

cudaError_t launch_schur64(const BatchView &bv, const ProblemParams &P, const float *C, const float *g, const float *c,
                           double *S64, double *gamma64, double *Ginv64c, int num_sms, cudaStream_t s, int ctas_per_sm)
{
    if (bv.total_knots <= 0) return cudaSuccess;
    if (!bv.st || !Ginv64c) return cudaErrorInvalidValue;
    int blocks = (bv.total_knots + S64_WARPS - 1) / S64_WARPS;
    const int cap = num_sms * ctas_per_sm;
    if (blocks > cap) blocks = cap;
    schur64_kernel<<<blocks, 32 * S64_WARPS, 0, s>>>(bv, P.qd_cost, P.r_cost, C, g, c, S64, gamma64, Ginv64c);
    return cudaGetLastError();
}

cudaError_t launch_schur64_gamma(const BatchView &bv, const double *S64, const double *Ginv64c, const float *C,
                                 const float *g, const float *c, double *gamma64, int num_sms, cudaStream_t s)
{
    if (bv.total_knots <= 0) return cudaSuccess;
    int blocks = (bv.total_knots + 3) / 4;
    if (blocks > num_sms * 16) blocks = num_sms * 16;
    schur64_gamma_kernel<<<blocks, 128, 0, s>>>(bv, S64, Ginv64c, C, g, c, gamma64);
    return cudaGetLastError();
}

}  // namespace gpt

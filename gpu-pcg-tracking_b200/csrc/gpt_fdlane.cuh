// gpt_fdlane.cuh -- forward dynamics and its gradient with one state per lane (32 states per warp): the throughput
// form of the half-warp evaluation in gpt_kkt.cu and gpt_grid.cu, which gives 16 lanes a state and has every lane
// repeat the value pass beside its tangent.  Here the value pass runs once per state and each tangent only through the
// links it reaches (direction j leaves the links before j at rest), about 600 instructions of a warp per state
// against 2150.  A warp takes some 20 us whatever the number of states, so the half-warp form stays the better one for
// few states.
//
// The formulas are that form's, in FP32 with the same FP64 elimination; the order of some sums differs, so the two
// agree to FP32 rounding.
//
// Per-lane state that a runtime index selects lives in shared memory, [item][lane].
#pragma once
#include "gpt_dyn.cuh"

namespace gpt {

constexpr int FL_V = 0, FL_IV = 6 * model::NJ, FL_XA = 12 * model::NJ, FL_F = 16 * model::NJ, FL_N = 20 * model::NJ;

struct FdLaneSmem {
    float base[FL_N][32];  // per link: v (6), I v (6), X a (entries 0, 1, 3, 4), accumulated f (the same entries)
    float Minv[CC][32];
    float out[NS * 34];    // a block of output rows on its way to memory (store_rows)
};

// ---- two FP32 values per operation (fma.rn.f32x2): the mass matrix's columns 2p, 2p + 1 and the tangents of q_d and
// qd_d run as the two halves
struct f2 {
    unsigned long long r;
};
__device__ __forceinline__ f2 pk2(float lo, float hi)
{
    f2 o;
    asm("mov.b64 %0, {%1, %2};" : "=l"(o.r) : "f"(lo), "f"(hi));
    return o;
}
__device__ __forceinline__ void un2(f2 a, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.r)); }
__device__ __forceinline__ f2 du2(float a) { return pk2(a, a); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 o;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(o.r) : "l"(a.r), "l"(b.r), "l"(c.r));
    return o;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 o;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(o.r) : "l"(a.r), "l"(b.r));
    return o;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 o;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(o.r) : "l"(a.r), "l"(b.r));
    return o;
}
__device__ __forceinline__ f2 neg2(f2 a)
{
    f2 o;
    o.r = a.r ^ 0x8000000080000000ull;
    return o;
}

// a joint's cos, sin and -sin (kind 1: -cos) in both halves
template <int J>
struct Rot2 {
    f2 c, s, n;
    __device__ __forceinline__ explicit Rot2(const JointTrig &t)
    {
        c = du2(t.c[J]);
        s = du2(t.s[J]);
        constexpr int K = model::kJointKind[J];
        n = du2(K == 1 ? -t.c[J] : -t.s[J]);
    }
    // E w (rot_apply) and E^T w (rot_apply_T)
    __device__ __forceinline__ void apply(const f2 *w, f2 *o) const
    {
        constexpr int K = model::kJointKind[J];
        if constexpr (K == 0) {
            o[0] = fma2(c, w[0], mul2(s, w[1]));
            o[1] = fma2(n, w[0], mul2(c, w[1]));
            o[2] = w[2];
        } else if constexpr (K == 1) {
            o[0] = fma2(n, w[0], mul2(s, w[2]));
            o[1] = fma2(s, w[0], mul2(c, w[2]));
            o[2] = w[1];
        } else {
            o[0] = fma2(c, w[0], mul2(s, w[2]));
            o[1] = fma2(n, w[0], mul2(c, w[2]));
            o[2] = neg2(w[1]);
        }
    }
    __device__ __forceinline__ void apply_T(const f2 *w, f2 *o) const
    {
        constexpr int K = model::kJointKind[J];
        if constexpr (K == 0) {
            o[0] = fma2(c, w[0], mul2(n, w[1]));
            o[1] = fma2(s, w[0], mul2(c, w[1]));
            o[2] = w[2];
        } else if constexpr (K == 1) {
            o[0] = fma2(n, w[0], mul2(s, w[1]));
            o[1] = w[2];
            o[2] = fma2(s, w[0], mul2(c, w[1]));
        } else {
            o[0] = fma2(c, w[0], mul2(n, w[1]));
            o[1] = neg2(w[2]);
            o[2] = fma2(s, w[0], mul2(c, w[1]));
        }
    }
    // motion transform parent -> child (xmot)
    __device__ __forceinline__ void motion(const f2 *m, f2 *o) const
    {
        constexpr float py = model::kJointP[J][1], pz = model::kJointP[J][2];
        f2 u[3] = {m[3], m[4], m[5]};
        if constexpr (py == 0.f) {
            u[0] = fma2(du2(pz), m[1], u[0]);
            u[1] = fma2(du2(-pz), m[0], u[1]);
        } else {
            u[0] = fma2(du2(-py), m[2], u[0]);
            u[2] = fma2(du2(py), m[0], u[2]);
        }
        f2 w[3] = {m[0], m[1], m[2]};
        apply(w, o);
        apply(u, o + 3);
    }
    // force transform child -> parent added to o (xforce_T)
    __device__ __forceinline__ void force_add(const f2 *f, f2 *o) const
    {
        constexpr float py = model::kJointP[J][1], pz = model::kJointP[J][2];
        f2 a[3], b[3];
        apply_T(f, a);
        apply_T(f + 3, b);
        if constexpr (py == 0.f) {
            a[0] = fma2(du2(-pz), b[1], a[0]);
            a[1] = fma2(du2(pz), b[0], a[1]);
        } else {
            a[0] = fma2(du2(py), b[2], a[0]);
            a[2] = fma2(du2(-py), b[0], a[2]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            o[k] = add2(o[k], a[k]);
            o[3 + k] = add2(o[3 + k], b[k]);
        }
    }
};

// acc + k w for a constant k, nothing for k = 0
__device__ __forceinline__ void cfma2(f2 &acc, float k, f2 w, bool &first)
{
    if (k == 0.f) return;
    acc = first ? mul2(du2(k), w) : fma2(du2(k), w, acc);
    first = false;
}
// spatial inertia of link J times a motion vector (inertia_apply)
template <int J>
__device__ __forceinline__ void inertia2(const f2 *v, f2 *o)
{
    constexpr float I[6] = {(float)model::ibar(J, 0), (float)model::ibar(J, 1), (float)model::ibar(J, 2),
                            (float)model::ibar(J, 3), (float)model::ibar(J, 4), (float)model::ibar(J, 5)};
    constexpr float m = (float)model::kMass[J];
    constexpr float cx = (float)(model::kMass[J] * model::kCom[J][0]), cy = (float)(model::kMass[J] * model::kCom[J][1]),
                    cz = (float)(model::kMass[J] * model::kCom[J][2]);
    constexpr float R[6][6] = {{I[0], I[3], I[4], 0.f, -cz, cy}, {I[3], I[1], I[5], cz, 0.f, -cx},
                               {I[4], I[5], I[2], -cy, cx, 0.f}, {0.f, cz, -cy, m, 0.f, 0.f},
                               {-cz, 0.f, cx, 0.f, m, 0.f},      {cy, -cx, 0.f, 0.f, 0.f, m}};
#pragma unroll
    for (int r = 0; r < 6; ++r) {
        bool first = true;
        o[r] = pk2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 6; ++k) cfma2(o[r], R[r][k], v[k], first);
    }
}
// o += a x_f b (crf), na = -a
__device__ __forceinline__ void crf2_add(const f2 *a, const f2 *na, const f2 *b, f2 *o)
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int i = (k + 1) % 3, j = (k + 2) % 3;
        o[k] = fma2(a[i], b[j], o[k]);
        o[k] = fma2(na[j], b[i], o[k]);
        o[k] = fma2(a[3 + i], b[3 + j], o[k]);
        o[k] = fma2(na[3 + j], b[3 + i], o[k]);
        o[3 + k] = fma2(a[i], b[3 + j], o[3 + k]);
        o[3 + k] = fma2(na[j], b[3 + i], o[3 + k]);
    }
}

// Columns 2p, 2p + 1 of the mass matrix, all rows (inverse dynamics at rest with a unit acceleration of the joint),
// into M[row + 7 column][lane]
template <int K>
__device__ __forceinline__ void fl_mcol_fwd(const JointTrig &t, int j, f2 (&a)[6], f2 (&f)[model::NJ][6])
{
    if (K >= j) {
        if (K > j) {
            f2 x[6];
            Rot2<K>(t).motion(a, x);
#pragma unroll
            for (int i = 0; i < 6; ++i) a[i] = x[i];
            if (K == j + 1) a[2] = add2(a[2], pk2(0.f, 1.f));
        }
        inertia2<K>(a, f[K]);
    } else {
#pragma unroll
        for (int i = 0; i < 6; ++i) f[K][i] = pk2(0.f, 0.f);
    }
    if constexpr (K + 1 < model::NJ) fl_mcol_fwd<K + 1>(t, j, a, f);
}
template <int K>
__device__ __forceinline__ void fl_force_bwd(const JointTrig &t, f2 (&f)[model::NJ][6])
{
    if constexpr (K > 0) {
        Rot2<K>(t).force_add(f[K], f[K - 1]);
        fl_force_bwd<K - 1>(t, f);
    }
}
__device__ __forceinline__ void fl_mass_matrix(const JointTrig &t, float (*M)[32], int lane)
{
#pragma unroll 1
    for (int j = 0; j < NQ; j += 2) {
        const f2 z = pk2(0.f, 0.f);
        f2 a[6] = {z, z, pk2(1.f, 0.f), z, z, z}, f[model::NJ][6];
        __syncthreads();
        fl_mcol_fwd<0>(t, j, a, f);
        fl_force_bwd<model::NJ - 1>(t, f);
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            float lo, hi;
            un2(f[k][2], lo, hi);
            M[k + NQ * j][lane] = lo;
            if (j + 1 < NQ) M[k + NQ * (j + 1)][lane] = hi;
        }
    }
}

// value pass at (q, qd, qdd): link quantities of the tangents into sm.base
template <int J>
__device__ __forceinline__ void fl_value_fwd(const JointTrig &t, const float (&qd)[NQ], const float (&qdd)[NQ],
                                             float (&vp)[6], float (&ap)[6], float (&f)[model::NJ][6], FdLaneSmem &sm,
                                             int lane)
{
    float Xv[6], Xa[6], cv[6], Iv[6], Ia[6], cIv[6];
    xmot<J>(t.c[J], t.s[J], vp, Xv);
    xmot<J>(t.c[J], t.s[J], ap, Xa);
#pragma unroll
    for (int k = 0; k < 6; ++k) vp[k] = Xv[k];
    vp[2] += qd[J];
    crm_s(vp, qd[J], cv);
#pragma unroll
    for (int k = 0; k < 6; ++k) ap[k] = Xa[k] + cv[k];
    ap[2] += qdd[J];
    inertia_apply<J>(vp, Iv);
    inertia_apply<J>(ap, Ia);
    crf(vp, Iv, cIv);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        f[J][k] = Ia[k] + cIv[k];
        sm.base[FL_V + 6 * J + k][lane] = vp[k];
        sm.base[FL_IV + 6 * J + k][lane] = Iv[k];
    }
    sm.base[FL_XA + 4 * J][lane] = Xa[0];
    sm.base[FL_XA + 4 * J + 1][lane] = Xa[1];
    sm.base[FL_XA + 4 * J + 2][lane] = Xa[3];
    sm.base[FL_XA + 4 * J + 3][lane] = Xa[4];
    if constexpr (J + 1 < model::NJ) fl_value_fwd<J + 1>(t, qd, qdd, vp, ap, f, sm, lane);
}
template <int J>
__device__ __forceinline__ void fl_value_bwd(const JointTrig &t, float (&f)[model::NJ][6], FdLaneSmem &sm, int lane)
{
    sm.base[FL_F + 4 * J][lane] = f[J][0];
    sm.base[FL_F + 4 * J + 1][lane] = f[J][1];
    sm.base[FL_F + 4 * J + 2][lane] = f[J][3];
    sm.base[FL_F + 4 * J + 3][lane] = f[J][4];
    if constexpr (J > 0) {
        float tf[6];
        xforce_T<J>(t.c[J], t.s[J], f[J], tf);
#pragma unroll
        for (int k = 0; k < 6; ++k) f[J - 1][k] += tf[k];
        fl_value_bwd<J - 1>(t, f, sm, lane);
    }
}

// Tangents of direction d, q_d in the low halves and qd_d in the high ones: links J .. 6 forward
template <int J>
__device__ __forceinline__ void fl_tangent_fwd(const JointTrig &t, const float (&qd)[NQ], int d, f2 (&dv)[6], f2 (&da)[6],
                                               f2 (&df)[model::NJ][6], const FdLaneSmem &sm, int lane)
{
    if (J >= d) {
        float v[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = sm.base[FL_V + 6 * J + k][lane];
        if (J > d) {
            const Rot2<J> rot(t);
            f2 x[6], y[6];
            rot.motion(dv, x);
            rot.motion(da, y);
            const f2 w = du2(qd[J]), n = du2(-qd[J]);
#pragma unroll
            for (int k = 0; k < 6; ++k) dv[k] = x[k];
            // + dv x S qd_J
            da[0] = fma2(dv[1], w, y[0]);
            da[1] = fma2(dv[0], n, y[1]);
            da[2] = y[2];
            da[3] = fma2(dv[4], w, y[3]);
            da[4] = fma2(dv[3], n, y[4]);
            da[5] = y[5];
        } else {
            // q_d: -S x (X v), -S x (X a) + dv x S qd_d (X v is v but for entry 2); qd_d: S, v x S
            const float xa0 = sm.base[FL_XA + 4 * J][lane], xa1 = sm.base[FL_XA + 4 * J + 1][lane],
                        xa3 = sm.base[FL_XA + 4 * J + 2][lane], xa4 = sm.base[FL_XA + 4 * J + 3][lane], w = qd[J];
            dv[0] = pk2(v[1], 0.f);
            dv[1] = pk2(-v[0], 0.f);
            dv[2] = pk2(0.f, 1.f);
            dv[3] = pk2(v[4], 0.f);
            dv[4] = pk2(-v[3], 0.f);
            dv[5] = pk2(0.f, 0.f);
            da[0] = pk2(fmaf(-v[0], w, xa1), v[1]);
            da[1] = pk2(-fmaf(v[1], w, xa0), -v[0]);
            da[2] = pk2(0.f, 0.f);
            da[3] = pk2(fmaf(-v[3], w, xa4), v[4]);
            da[4] = pk2(-fmaf(v[4], w, xa3), -v[3]);
            da[5] = pk2(0.f, 0.f);
        }
        f2 Idv[6], n[6], b[6];
        inertia2<J>(da, df[J]);
        inertia2<J>(dv, Idv);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            n[k] = neg2(dv[k]);
            b[k] = du2(sm.base[FL_IV + 6 * J + k][lane]);
        }
        crf2_add(dv, n, b, df[J]);  // dv x I v
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            b[k] = du2(v[k]);
            n[k] = du2(-v[k]);
        }
        crf2_add(b, n, Idv, df[J]);  // v x I dv
    } else {
#pragma unroll
        for (int k = 0; k < 6; ++k) df[J][k] = pk2(0.f, 0.f);
    }
    if constexpr (J + 1 < model::NJ) fl_tangent_fwd<J + 1>(t, qd, d, dv, da, df, sm, lane);
}
template <int J>
__device__ __forceinline__ void fl_tangent_bwd(const JointTrig &t, int d, f2 (&df)[model::NJ][6], const FdLaneSmem &sm,
                                               int lane)
{
    if constexpr (J > 0) {
        f2 f[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) f[k] = df[J][k];
        if (J == d) {  // q_d also turns the force that link d hands down: S x f
            f[0] = add2(f[0], pk2(-sm.base[FL_F + 4 * J + 1][lane], 0.f));
            f[1] = add2(f[1], pk2(sm.base[FL_F + 4 * J][lane], 0.f));
            f[3] = add2(f[3], pk2(-sm.base[FL_F + 4 * J + 3][lane], 0.f));
            f[4] = add2(f[4], pk2(sm.base[FL_F + 4 * J + 2][lane], 0.f));
        }
        Rot2<J>(t).force_add(f, df[J - 1]);
        fl_tangent_bwd<J - 1>(t, d, df, sm, lane);
    }
}
// a block of df/du's columns: d/dq, d/dqd, d/du
template <int I>
struct FdBlock {
    static constexpr int block = I;
};

// The CTA's warps take the directions together (the barrier): the loop's code then comes from the instruction cache once
// for the warps of a scheduler instead of once for each, which is what bounds the kernel.
template <class Emit>
__device__ __forceinline__ void fl_directions(const JointTrig &t, const float (&qd)[NQ], const FdLaneSmem &sm, int lane,
                                              Emit emit)
{
#pragma unroll 1
    for (int d = 0; d < NQ; ++d) {
        f2 dv[6], da[6], df[model::NJ][6];
#pragma unroll
        for (int k = 0; k < 6; ++k) dv[k] = da[k] = pk2(0.f, 0.f);
        __syncthreads();
        fl_tangent_fwd<0>(t, qd, d, dv, da, df, sm, lane);
        fl_tangent_bwd<model::NJ - 1>(t, d, df, sm, lane);
        float lo[NQ], hi[NQ];
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            f2 acc = pk2(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < NQ; ++k) acc = fma2(du2(sm.Minv[r + NQ * k][lane]), df[k][2], acc);
            un2(neg2(acc), lo[r], hi[r]);
        }
        emit(FdBlock<0>(), d, lo);
        emit(FdBlock<1>(), d, hi);
    }
}

// qdd = M^{-1} (u - c) alone: the FP64 L D L^T of M's symmetric part, without pivoting (M is positive definite)
__device__ __forceinline__ void fd_lane(const JointTrig &t, const float (&qd)[NQ], const float (&u)[NC], float (&qdd)[NQ],
                                        float (*M)[32], int lane)
{
    double A[NQ][NQ], x[NQ], rd[NQ];
    {
        float zero[NQ], c[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) zero[i] = 0.f;
        fl_mass_matrix(t, M, lane);
        rnea<false>(t, qd, zero, -1, -1, c, nullptr);
#pragma unroll
        for (int j = 0; j < NQ; ++j) {
#pragma unroll
            for (int r = j; r < NQ; ++r) A[j][r] = 0.5 * ((double)M[r + NQ * j][lane] + (double)M[j + NQ * r][lane]);
            x[j] = (double)u[j] - (double)c[j];
        }
    }
#pragma unroll
    for (int p = 0; p < NQ; ++p) {
        rd[p] = rcp_newton(A[p][p]);
#pragma unroll
        for (int i = p + 1; i < NQ; ++i) {
            const double l = A[p][i] * rd[p];
            x[i] = fma(-l, x[p], x[i]);
#pragma unroll
            for (int r = i; r < NQ; ++r) A[i][r] = fma(-l, A[p][r], A[i][r]);
        }
    }
#pragma unroll
    for (int p = NQ - 1; p >= 0; --p) {
#pragma unroll
        for (int i = p + 1; i < NQ; ++i) x[p] = fma(-A[p][i], x[i], x[p]);
        x[p] *= rd[p];
        qdd[p] = (float)x[p];
    }
}

// qdd = M^{-1} (u - c) and the columns of df/du = [-M^{-1} dID/dq, -M^{-1} dID/dqd, M^{-1}] at (q, qd, u), each handed to
// emit(FdBlock<i>(), column of the block, values[7]) by every lane at the same time
template <class Emit>
__device__ __forceinline__ void fd_gradient_lane(const JointTrig &t, const float (&qd)[NQ], const float (&u)[NC],
                                                 float (&qdd)[NQ], FdLaneSmem &sm, int lane, Emit emit)
{
    {
        // [M | u - c] in FP64 (M's symmetric part), the inverse in place by Gauss-Jordan without pivoting
        double A[NQ][NQ], rhs[NQ];
        {
            float zero[NQ], c[NQ];
#pragma unroll
            for (int i = 0; i < NQ; ++i) zero[i] = 0.f;
            fl_mass_matrix(t, sm.Minv, lane);
            rnea<false>(t, qd, zero, -1, -1, c, nullptr);
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
#pragma unroll
                for (int r = 0; r < NQ; ++r)
                    A[j][r] = 0.5 * ((double)sm.Minv[r + NQ * j][lane] + (double)sm.Minv[j + NQ * r][lane]);
                rhs[j] = (double)u[j] - (double)c[j];
            }
        }
#pragma unroll
        for (int p = 0; p < NQ; ++p) {
            const double r = rcp_newton(A[p][p]);
            double pc[NQ];  // the pivot column
#pragma unroll
            for (int i = 0; i < NQ; ++i) pc[i] = A[p][i];
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const double prow = j == p ? r : A[j][p] * r;
#pragma unroll
                for (int i = 0; i < NQ; ++i)
                    if (i != p) A[j][i] = j == p ? -pc[i] * prow : fma(-pc[i], prow, A[j][i]);
                A[j][p] = prow;
            }
            const double prow = rhs[p] * r;
#pragma unroll
            for (int i = 0; i < NQ; ++i)
                if (i != p) rhs[i] = fma(-pc[i], prow, rhs[i]);
            rhs[p] = prow;
        }
#pragma unroll
        for (int j = 0; j < NQ; ++j) {
            qdd[j] = (float)rhs[j];
#pragma unroll
            for (int r = 0; r < NQ; ++r) sm.Minv[r + NQ * j][lane] = (float)A[j][r];
        }
    }
    {
        float vp[6], ap[6], f[model::NJ][6];
#pragma unroll
        for (int k = 0; k < 6; ++k) vp[k] = ap[k] = 0.f;
        fl_value_fwd<0>(t, qd, qdd, vp, ap, f, sm, lane);
        fl_value_bwd<model::NJ - 1>(t, f, sm, lane);
    }
    fl_directions(t, qd, sm, lane, emit);
#pragma unroll 1
    for (int j = 0; j < NC; ++j) {
        float col[NQ];
#pragma unroll
        for (int r = 0; r < NQ; ++r) col[r] = sm.Minv[r + NQ * j][lane];
        emit(FdBlock<2>(), j, col);
    }
}

// Store R values per lane (v[0 .. R-1] of state i = lane) as R consecutive floats at dst + STRIDE i for the lanes in
// mask; every lane calls it.  Through shared memory, 32 / R states by R lanes at a time: a store then covers that many
// contiguous runs, its addresses differ from the last one's by a constant, and neither side has bank conflicts.
template <int R, int STRIDE>
__device__ __forceinline__ void store_rows(float (&buf)[NS * 34], const float (&v)[R], float *dst, uint32_t mask, int lane)
{
    constexpr int K = 32 / R, PITCH = 32 + K;
    static_assert(R * PITCH <= NS * 34 && 32 % K == 0, "the buffer");
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) buf[PITCH * r + lane] = v[r];
    __syncwarp();
    const int k = lane / R, r = lane - R * k;
    if (k < K) {
        const float *src = buf + PITCH * r + k;
        dst += STRIDE * k + r;
        mask >>= k;
#pragma unroll
        for (int i = 0; i < 32; i += K)
            if (mask >> i & 1u) dst[(ptrdiff_t)STRIDE * i] = src[i];
    }
}

}  // namespace gpt

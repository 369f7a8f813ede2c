// gpt_part.cu -- the partitioned PCG (pcg_cluster_size PCG_WARP_QUAD): one CTA or one cluster of CTAs per
// instance, whose warps factor parts of the horizon.
//
// Solves S lambda = gamma by conjugate gradients with the exact inverse of S as the preconditioner
// (z = S^{-1} r up to rounding), so the iteration stops after one step, from any start.  It starts from lambda = 0
// (r_0 = gamma); asked to start from the given lambda, it keeps one that meets the tolerance (warm).  With M = -S (SPD),
// A_k = M_kk and E_k = M_{k,k-1} = -L_k (L_k the left block of row k of S), the horizon is cut by P - 1 separator
// knots s_1 < ... < s_{P-1} into P parts.  Part 0 is eliminated top-down toward s_1 and part P-1
// bottom-up toward s_{P-1}; a middle part top-down from its left to its right separator, which couples
// the two.  The separators' block-tridiagonal system is eliminated by two warps from both ends, then every
// part is solved backward.  This is the block L D L^T of M with the parts' knots ordered before the
// separators.
//
// One elimination step (part_step) is the symmetric elimination of the 14 unknowns of one knot from
//   [ D  E^T | y  ]      D: the knot's block, y its right-hand side,
//   [ E  A'  | y' ]      A', y': the next knot's (E its coupling),
// with D = L B L^T, B block diagonal with the 2 x 2 pivots {2t, 2t+1}, L unit block lower: seven block
// pivots turn [D | E^T | y] into [. | W | z] = L^{-1} [E^T | y], and the next knot's block and
// right-hand side are A' - W^T B^{-1} W and y' - W^T B^{-1} z.  Lane pair (c, h) = (lane >> 1, lane & 1)
// holds the rows i = 2q + h (q < 7) of column c; column 14 of the E^T set carries y.  The registers
// of a finished column of D collect that column of L^{-1}.  A middle part also carries F_k = M_{k, left
// separator}: with V = L^{-1} F_k the next knot's F is -W^T B^{-1} V, and the left separator's update
// -V^T B^{-1} [V, z].  L^{-1}, with B^{-1} in its diagonal blocks, is stored for the backward solve
//   x_k = L^{-T} B^{-1} (z_k + L^{-1} t),  t = -E^T x_next - F_k x_left.
// The pivots run on the FP64 pipe with the pivot rows broadcast through shared memory; the rank-14
// products of a middle part on the FP64 tensor cores (part_step_mid).  What bounds a step is the length of its
// dependent chain and the instructions around it: at 512 x 128 issue is 0.41 per cycle and scheduler, the FP64
// pipe 23 % and the L1 and shared-memory pipe 66 % busy (ncu).
//
// A preconditioner application is one such factorisation: with an exact preconditioner the iteration
// almost always ends after the first, so nothing but L^{-1} and F is kept for another right-hand side.
//
// The backward sweep forms S x as it goes (it reads the rows of S for their coupling blocks anyway): the CG
// iteration's S p is its negative.
//
// Storage per knot: QW_STRIDE doubles of the FP64 workspace: L^{-1} (QINV), F_k row-major (SS), S x, and,
// only when the iteration goes on, the CG vectors.  S is read from global memory in rows staged by
// cp.async.
#include <cooperative_groups.h>

#include <type_traits>

#include "gpt_common.cuh"
#include "gpt_internal.h"
#include "gpt_layout.h"

namespace cg = cooperative_groups;

namespace gpt {

constexpr int PK_LEFT_N = SS, PK_TRI = 105;
constexpr int QW_STRIDE = 2 * SS;  // workspace doubles per knot
// L^{-1} of a knot: entry (i, c), i >= c, at 2 q (q + 1) + 2 c + h with q = i >> 1, h = i & 1: the lanes'
// register q contiguous over the lanes (one hole per q, so 112 slots for the 105 entries)
constexpr int QINV = 112;
constexpr int QW_F = QINV, QW_RES = QINV + SS, QW_LAM = QW_RES + NS, QW_P = QW_LAM + NS, QW_V = QW_P + NS,
              QW_SX = QW_V + NS;
static_assert(QW_SX + NS <= QW_STRIDE, "the CG vectors fit the knot's workspace");
constexpr int QROW_D = PK64;               // a staged row of S (FP64)
constexpr int QBACK_D = QINV + QROW_D;     // a staged step of the backward sweep: L^{-1} and a row of S
constexpr int QSLOT_D = 308;               // a staging slot of the walk (two slots of the sweep in three)
constexpr int QSEP = 7 * 32;               // a lane-layout block (7 registers x 32 lanes)
static_assert(3 * QSEP <= 3 * QSLOT_D && 2 * QBACK_D <= 3 * QSLOT_D && QROW_D <= QSLOT_D,
              "the separators' blocks and two steps of the sweep fit three slots");
constexpr int QLD = 20;                    // leading dimension of W and V (conflict-free fragment loads)
constexpr int QW_D = NS * QLD;             // W or V (14 rows x 16 columns)
constexpr int QROWS_D = 2 * 2 * 37;        // pivot rows: 2 sets of 2 rows (D, E^T), 37 pairs apart
constexpr int QBUF = QROWS_D + 2 * NS;     // pivot rows; B^{-1} by rows
constexpr int RED_N = 3;                   // values of a reduction, and one more apart from them (the start's check)
constexpr int RR_PERIOD = 32;              // CG iterations between true-residual replacements

// A kernel variant: a cluster of CL CTAs of WC warps per instance (NW = CL WC parts, in order over the CTAs), SL staging
// slots per warp, MINB CTAs per SM, EDGE the length of an edge part in tenths of a middle part's
template <int CL_, int WC_, int SL_, int MINB_, int EDGE_>
struct PartCfg {
    static_assert(WC_ >= 2 && SL_ >= 3, "two warps, three slots at least");
    static constexpr int CL = CL_, WC = WC_, NW = CL * WC, SL = SL_, MINB = MINB_, EDGE = EDGE_;
    static constexpr int REGION = SL * QSLOT_D;
    static constexpr int SB = REGION / QBACK_D;  // slots of the backward sweep
    // the middle parts' W; after the walks the separators' L^{-1}, the bottom half's update of the middle one and the
    // terms of S x that belong to a separator
    static constexpr int MIDS = CL == 1 ? NW - 2 : WC;
    static constexpr int SEP_B = (NW - 1) * QINV, SEP_SX = SEP_B + (NW > 2 ? QSEP : 0);
    static constexpr int MID = MIDS * QW_D > SEP_SX + WC * NS ? MIDS * QW_D : SEP_SX + WC * NS;
    static size_t smem_bytes(int n)
    {
        return sizeof(double) * (size_t)(NS * n + WC * (REGION + QBUF) + MID + 2 * NW * (RED_N + 1) + 4);
    }
};

__device__ __forceinline__ int tri_idx(int r, int c)  // packed lower triangle, any order
{
    return r >= c ? ((r * (r + 1)) >> 1) + c : ((c * (c + 1)) >> 1) + r;
}
__device__ __forceinline__ int inv_idx(int i, int c) { return 2 * (i >> 1) * ((i >> 1) + 1) + 2 * c + (i & 1); }

// rows 2t, 2t + 1 (v0, v1) of a column, from this lane's own row and its partner's
__device__ __forceinline__ void pair_rows(double own, double other, int h, double &v0, double &v1)
{
    v0 = h ? other : own;
    v1 = h ? own : other;
}

// One elimination step on the lane layout above.  In: a = D (columns 14, 15: anything finite), e = [E^T | y | 0],
// b = [A' | y' | 0].  Out: a = L^{-1} with the 2 x 2 blocks of B^{-1} on its diagonal (lower part), e = [W | z],
// b -= W^T B^{-1} [W | z].  buf: QROWS_D doubles.  Seven block pivots of about 120 cycles each when the warp
// is alone on its scheduler (the chain of two shared-memory trips and a reciprocal).
__device__ __forceinline__ void part_step(double (&a)[7], double (&e)[7], double (&b)[7], double *buf, int lane)
{
    const int c = lane >> 1, h = lane & 1;
    // the pivot rows: (D, E^T) pairs, column c at place 9 (c & 1) + (c >> 1), so that lane half h reads rows
    // 2q + h at 9 h + q without bank conflicts
    const int pos = 9 * (c & 1) + (c >> 1);
    double2 *rows = reinterpret_cast<double2 *>(buf);
#pragma unroll
    for (int t = 0; t < 7; ++t) {
        double2 *bk = rows + (t & 1) * 37;
        bk[18 * h + pos] = make_double2(a[t], e[t]);
        __syncwarp();
        const double x = bk[t].x, y = bk[9 + t].x, z = bk[27 + t].x;  // the pivot block
        const double2 op = bk[18 * (h ^ 1) + pos];
        const double rd = rcp_cubic(fma(x, z, -y * y));
        const double i00 = z * rd, i01 = -y * rd, i11 = x * rd;
        const bool p0 = c == 2 * t, p1 = c == 2 * t + 1, piv = p0 || p1;
        // this column's pivot rows (the identity's in the pivot columns) times B^{-1}
        double v0, v1, w0, w1;
        pair_rows(a[t], op.x, h, v0, v1);
        pair_rows(e[t], op.y, h, w0, w1);
        v0 = piv ? (p0 ? 1.0 : 0.0) : v0;
        v1 = piv ? (p1 ? 1.0 : 0.0) : v1;
        const double n0 = fma(i00, v0, i01 * v1), n1 = fma(i01, v0, i11 * v1);
        const double m0 = fma(i00, w0, i01 * w1), m1 = fma(i01, w0, i11 * w1);
        const int keep = piv ? 0 : -1;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const double2 r0 = bk[9 * h + q], r1 = bk[18 + 9 * h + q];
            if (q > t) {
                const double av = __hiloint2double(__double2hiint(a[q]) & keep, __double2loint(a[q]) & keep);
                a[q] = fma(-r0.x, n0, fma(-r1.x, n1, av));
                e[q] = fma(-r0.x, m0, fma(-r1.x, m1, e[q]));
            }
            b[q] = fma(-r0.y, m0, fma(-r1.y, m1, b[q]));
        }
        const double dv = p0 ? (h ? i01 : i00) : i11;
        a[t] = piv ? dv : a[t];
    }
}

// The same for a middle part, with f = F (0 in columns 14, 15): b = -W^T B^{-1} [W | z] (not added to the next
// block), f = -W^T B^{-1} V, acc -= V^T B^{-1} [V | z] (tiles (0,0), (0,1), (1,1) of the tensor-core layout).  The
// three products run on the FP64 tensor cores after the pivots: lane by lane they need 294 more FP64
// instructions and 28 more live registers than the kernel has (measured, 16 warps per SM: 7.2 k cycles
// a step lane by lane, 5.7 k this way).  buf: QROWS_D + 28 doubles; W and vbuf QW_D each.
__device__ __forceinline__ void part_step_mid(double (&a)[7], double (&e)[7], double (&f)[7], double (&b)[7],
                                              double (&acc)[3][2], double *buf, double *W, double *vbuf, int lane)
{
    const int c = lane >> 1, h = lane & 1;
    const int pos = 8 * (c & 1) + (c >> 1);  // a row of D: lane half h reads rows 2q + h at 8 h + q
    double *binv = buf + QROWS_D;
#pragma unroll
    for (int t = 0; t < 7; ++t) {
        double *bk = buf + (t & 1) * 32;
        bk[16 * h + pos] = a[t];
        W[(2 * t + h) * QLD + c] = e[t];
        vbuf[(2 * t + h) * QLD + c] = f[t];
        __syncwarp();
        const double x = bk[t], y = bk[8 + t], z = bk[24 + t];
        const double ap = bk[16 * (h ^ 1) + pos], ep = W[(2 * t + (h ^ 1)) * QLD + c],
                     fp = vbuf[(2 * t + (h ^ 1)) * QLD + c];
        const double rd = rcp_cubic(fma(x, z, -y * y));
        const double i00 = z * rd, i01 = -y * rd, i11 = x * rd;
        if (c == 0) *reinterpret_cast<double2 *>(binv + 2 * (2 * t + h)) = make_double2(h ? i11 : i00, i01);
        const bool p0 = c == 2 * t, p1 = c == 2 * t + 1, piv = p0 || p1;
        double v0, v1, w0, w1, g0, g1;
        pair_rows(a[t], ap, h, v0, v1);
        pair_rows(e[t], ep, h, w0, w1);
        pair_rows(f[t], fp, h, g0, g1);
        v0 = piv ? (p0 ? 1.0 : 0.0) : v0;
        v1 = piv ? (p1 ? 1.0 : 0.0) : v1;
        const double n0 = fma(i00, v0, i01 * v1), n1 = fma(i01, v0, i11 * v1);
        const double m0 = fma(i00, w0, i01 * w1), m1 = fma(i01, w0, i11 * w1);
        const double s0 = fma(i00, g0, i01 * g1), s1 = fma(i01, g0, i11 * g1);
        const int keep = piv ? 0 : -1;
#pragma unroll
        for (int j = (t + 1) >> 1; j < 4; ++j) {
            const double2 u0 = *reinterpret_cast<const double2 *>(bk + 8 * h + 2 * j);
            const double2 u1 = *reinterpret_cast<const double2 *>(bk + 16 + 8 * h + 2 * j);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int q = 2 * j + k;
                if (q <= t || q > 6) continue;
                const double r0 = k ? u0.y : u0.x, r1 = k ? u1.y : u1.x;
                const double av = __hiloint2double(__double2hiint(a[q]) & keep, __double2loint(a[q]) & keep);
                a[q] = fma(-r0, n0, fma(-r1, n1, av));
                e[q] = fma(-r0, m0, fma(-r1, m1, e[q]));
                f[q] = fma(-r0, s0, fma(-r1, s1, f[q]));
            }
        }
        const double dv = p0 ? (h ? i01 : i00) : i11;
        a[t] = piv ? dv : a[t];
    }
    __syncwarp();
    // rows k of W and V in chunks of four: fragments X_I = X(4 kk + t, 8 I + g), scaled by B^{-1} (row k's partner in
    // its 2 x 2 block is in lane t ^ 1)
    const int g = lane >> 2, t = lane & 3;
    double cb[3][2] = {}, cf[2][2][2] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        const bool in = kk < 3 || t < 2;
        const int k = in ? 4 * kk + t : 0;
        double w[2], v[2], y[2], s[2];
        const double2 bi = *reinterpret_cast<const double2 *>(binv + 2 * k);
        const double id = in ? bi.x : 0.0, io = in ? bi.y : 0.0;
#pragma unroll
        for (int I = 0; I < 2; ++I) {
            w[I] = W[k * QLD + 8 * I + g];
            v[I] = vbuf[k * QLD + 8 * I + g];
            y[I] = -fma(id, w[I], io * __shfl_xor_sync(0xffffffffu, w[I], 1));
            s[I] = -fma(id, v[I], io * __shfl_xor_sync(0xffffffffu, v[I], 1));
        }
        const double s1 = g == 6 ? y[1] : s[1];  // column 14: z
        mma884_f64(cb[0], w[0], y[0]);
        mma884_f64(cb[1], w[0], y[1]);
        mma884_f64(cb[2], w[1], y[1]);
#pragma unroll
        for (int I = 0; I < 2; ++I)
#pragma unroll
            for (int J = 0; J < 2; ++J) mma884_f64(cf[I][J], w[I], s[J]);
        mma884_f64(acc[0], v[0], s[0]);
        mma884_f64(acc[1], v[0], s1);
        mma884_f64(acc[2], v[1], s1);
    }
    __syncwarp();
    // back to the lane layout through W and V: element (i, j) at i QLD + j
    auto put2 = [&](double *d, int i, int j, const double (&v)[2]) {
        *reinterpret_cast<double2 *>(d + i * QLD + j) = make_double2(v[0], v[1]);
    };
    put2(W, g, 2 * t, cb[0]);
    put2(W, g, 8 + 2 * t, cb[1]);
    put2(vbuf, g, 2 * t, cf[0][0]);
    put2(vbuf, g, 8 + 2 * t, cf[0][1]);
    if (g < 6) {
        put2(W, 8 + g, 8 + 2 * t, cb[2]);
        put2(vbuf, 8 + g, 2 * t, cf[1][0]);
        put2(vbuf, 8 + g, 8 + 2 * t, cf[1][1]);
    }
    if (t < 3) {  // the lower off-diagonal tile by symmetry
        W[(8 + 2 * t) * QLD + g] = cb[1][0];
        W[(9 + 2 * t) * QLD + g] = cb[1][1];
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        b[q] = W[(2 * q + h) * QLD + c];
        f[q] = vbuf[(2 * q + h) * QLD + c];
    }
}

// The backward solve of one knot on a warp.  Its L^{-1} and B^{-1} entries are loaded ahead of the step that needs
// them (load), which takes the coupling term t (both lanes of pair c) and overwrites the knot's z at zk by x; sc: 28
// doubles of scratch.
struct PartBack {
    double row[7], col[7], id, io;
    __device__ __forceinline__ void load(const double *inv, int lane)
    {
        const int c = lane >> 1, h = lane & 1, cc = c < NS ? c : NS - 1, blk = cc & ~1;
        const double *pr = inv + inv_idx(cc, h), *pc = inv + 2 * cc + h;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const int j = 2 * q + h;
            const double rv = pr[4 * q], cv = pc[2 * q * (q + 1)];
            row[q] = j < blk ? rv : 0.0;
            col[q] = j > blk + 1 ? cv : 0.0;
        }
        id = inv[inv_idx(cc, cc)];
        io = inv[inv_idx(blk + 1, blk)];
    }
    __device__ __forceinline__ void step(double t, double *zk, double *sc, int lane) const
    {
        const int c = lane >> 1, h = lane & 1, cc = c < NS ? c : NS - 1;
        const bool wr = h == 0 && c < NS;
        const double z = zk[cc];
        if (wr) sc[c] = t;
        __syncwarp();
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int q = 0; q < 7; ++q) (q & 1 ? s1 : s0) = fma(row[q], sc[2 * q + h], q & 1 ? s1 : s0);
        s0 += s1;
        s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
        const double u = (z + t) + s0;
        const double w = fma(id, u, io * __shfl_xor_sync(0xffffffffu, u, 2));
        if (wr) sc[NS + c] = w;
        __syncwarp();
        s0 = s1 = 0.0;
#pragma unroll
        for (int q = 0; q < 7; ++q) (q & 1 ? s1 : s0) = fma(col[q], sc[NS + 2 * q + h], q & 1 ? s1 : s0);
        s0 += s1;
        s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
        if (wr) zk[c] = w + s0;
        __syncwarp();
    }
};

// the lanes of a warp copy CHUNKS 16-byte chunks (both addresses 16-byte aligned)
template <int CHUNKS>
__device__ __forceinline__ void warp_stage(void *sdst, const void *gsrc, int lane)
{
    char *d = reinterpret_cast<char *>(sdst) + 16 * lane;
    const char *g = reinterpret_cast<const char *>(gsrc) + 16 * lane;
#pragma unroll
    for (int i = 0; i < CHUNKS; i += 32)
        if (i + 32 <= CHUNKS || lane < CHUNKS - i) cp_async16(d + 16 * i, g + 16 * i);
}

template <int FMT>
struct PartRows {
    using ST = typename std::conditional<FMT == 2, double, float>::type;
    static constexpr int ROW_CHUNKS = (PK_LEFT_N + PK_TRI) * (int)sizeof(ST) / 16 + 1;  // a row of S, 16-byte chunks
    static_assert(ROW_CHUNKS * 16 <= (FMT == 2 ? PK64 : PK) * (int)sizeof(ST) && ROW_CHUNKS * 16 <= QROW_D * 8,
                  "a staged row fits its slot and its row of S");
};

// Shared memory of a CTA
template <class CF>
struct PartSmem {
    double *stg, *buf, *wmid, *red, *xv;
    int *lay;
    __device__ __forceinline__ explicit PartSmem(double *base)
    {
        stg = base;                         // per warp: staged rows / steps; the separators' blocks
        buf = stg + CF::WC * CF::REGION;    // per warp: pivot rows; the backward sweep's scratch
        wmid = buf + CF::WC * QBUF;
        red = wmid + CF::MID;               // 2 sets x NW warps x RED_N, 2 sets x NW warps
        lay = reinterpret_cast<int *>(red + 2 * CF::NW * (RED_N + 1));  // parts, first separator, spacing, this CTA's knots
        xv = red + 2 * CF::NW * (RED_N + 1) + 4;  // 14 n: y, then z, then x (of the CTA's knots and all separators)
    }
};

// barrier over the instance's threads
template <class CF>
__device__ __forceinline__ void part_sync()
{
    if constexpr (CF::CL == 1) __syncthreads();
    else cg::this_cluster().sync();
}
template <class CF>
__device__ __forceinline__ int part_rank()
{
    if constexpr (CF::CL == 1) return 0;
    else return (int)cg::this_cluster().block_rank();
}
// address p of this CTA's shared memory in CTA r of the cluster
template <class CF>
__device__ __forceinline__ double *part_peer(double *p, int r)
{
    if constexpr (CF::CL == 1) return p;
    else return cg::this_cluster().map_shared_rank(p, r);
}

// The elimination of one part (knots pa .. pb; SPK: a middle part) by the calling warp: L^{-1} (and F) of
// every knot into the workspace, z into xv, and into the warp's staging region, in the lane layout, its
// separators' blocks: [0] top-down the right separator's [block | y], bottom-up the left one's update; SPK:
// [1] the left separator's update, [2] the coupling of the right separator to the left one.
template <int FMT, class CF, bool SPK>
__device__ __forceinline__ void walk_part(const typename std::conditional<FMT == 2, double, float>::type *Sb, double *wsb,
                                       int pa, int pb, bool top, bool sep)
{
    using ST = typename std::conditional<FMT == 2, double, float>::type;
    constexpr size_t ks = FMT == 2 ? PK64 : PK;
    constexpr int ROW_CHUNKS = PartRows<FMT>::ROW_CHUNKS;
    extern __shared__ __align__(16) double part_dyn_smem[];
    const PartSmem<CF> ps(part_dyn_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = lane >> 1, h = lane & 1, cl = c < NS ? c : NS - 1;
    double *stg = ps.stg + warp * CF::REGION, *buf = ps.buf + warp * QBUF, *xv = ps.xv;
    double a[7], e[7], b[7], f[7], acc[3][2] = {};
    const int len = pb >= pa ? pb - pa + 1 : 0;
    const int k0 = top ? pa : pb, dir = top ? 1 : -1;
    const int nrows = top && sep ? len + 1 : len;  // top-down: the separator's row too
    const ST *src = Sb + (ptrdiff_t)ks * k0;
    const ptrdiff_t dsrc = top ? (ptrdiff_t)ks : -(ptrdiff_t)ks;
    auto stage = [&](int i, double *slot) {
        if (i < nrows) warp_stage<ROW_CHUNKS>(slot, src + dsrc * i, lane);
        cp_async_commit();
    };
    // [A' | y' | 0] of knot k from its row
    const double sgn = c < NS ? -1.0 : (c == NS ? 1.0 : 0.0);
    int tri[7];
#pragma unroll
    for (int q = 0; q < 7; ++q) tri[q] = PK_LEFT_N + tri_idx(2 * q + h, cl);
    auto ld_block = [&](const double *slot, int k, double (&v)[7]) {
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const double dv = (double)reinterpret_cast<const ST *>(slot)[tri[q]], yv = xv[NS * k + 2 * q + h];
            v[q] = sgn * (c < NS ? dv : yv);
        }
    };
    const int eo = top ? cl + NS * h : h + NS * cl, es = top ? 2 * NS : 2;  // E^T = -L^T or -L
    double *s0 = stg, *s1 = stg + QROW_D, *s2 = stg + 2 * QROW_D;           // rows st, st + 1, st + 2
    stage(0, s0);
    stage(1, s1);
    cp_async_wait<0>();
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        b[q] = f[q] = 0.0;
        if (SPK && c < NS) f[q] = -(double)reinterpret_cast<const ST *>(s0)[2 * q + h + NS * cl];  // F_a = -L_a
    }
    if (nrows > 0) ld_block(s0, k0, b);
    double *wk = wsb + (ptrdiff_t)k0 * QW_STRIDE + lane, *zk = xv + NS * k0 + h;
    for (int st = 0; st < len; ++st) {
        const bool more = st + 1 < nrows;
        const ST *er = reinterpret_cast<const ST *>(top ? s1 : s0) + eo;
        __syncwarp();  // s2 has been read
        stage(st + 2, s2);
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const double ev = (double)er[es * q];
            a[q] = b[q];
            e[q] = c < NS ? -ev : b[q];
        }
        if constexpr (SPK) {
            double *wf = wk - lane + QW_F + NS * h + c;
            if (c < NS) {
#pragma unroll
                for (int q = 0; q < 7; ++q) wf[28 * q] = f[q];
            }
            // row st is done with: its slot holds V
            part_step_mid(a, e, f, b, acc, buf, ps.wmid + (CF::CL == 1 ? warp - 1 : warp) * QW_D, s0, lane);
            double d[7];
            ld_block(s1, k0 + st + 1, d);  // a middle part ends at a separator: the next row exists
#pragma unroll
            for (int q = 0; q < 7; ++q) b[q] += d[q];
        } else {
            ld_block(s1, more ? k0 + dir * (st + 1) : 0, b);
            if (!more) {  // the walk's last knot: no next block, and top-down no coupling
#pragma unroll
                for (int q = 0; q < 7; ++q) {
                    b[q] = 0.0;
                    if (top && c < NS) e[q] = 0.0;
                }
            }
            part_step(a, e, b, buf, lane);
        }
#pragma unroll
        for (int q = 0; q < 7; ++q)
            if (c <= 2 * q + h && c < NS) wk[2 * q * (q + 1)] = a[q];
        if (c == NS) {
#pragma unroll
            for (int q = 0; q < 7; ++q) zk[2 * q] = e[q];
        }
        cp_async_wait<0>();  // row st + 2
        wk += top ? QW_STRIDE : -QW_STRIDE;
        zk += top ? NS : -NS;
        double *sx = s0;
        s0 = s1;
        s1 = s2;
        s2 = sx;
    }
    __syncwarp();
    // b: the right separator's block and y (top-down), or the update of the left one (bottom-up)
#pragma unroll
    for (int q = 0; q < 7; ++q) stg[32 * q + lane] = (top || len > 0) ? b[q] : 0.0;
    if constexpr (SPK) {
        const int g = lane >> 2, t = lane & 3;
        auto put = [&](int i, int j, double v) {
            if (i < NS && j <= NS) stg[QSEP + 32 * (i >> 1) + 2 * j + (i & 1)] = v;
        };
#pragma unroll
        for (int q = 0; q < 7; ++q) stg[2 * QSEP + 32 * q + lane] = f[q];  // M_{right separator, left one}
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            put(g, 2 * t + x, acc[0][x]);
            put(g, 8 + 2 * t + x, acc[1][x]);
            put(8 + g, 8 + 2 * t + x, acc[2][x]);
            if (8 + 2 * t + x < NS) put(8 + 2 * t + x, g, acc[1][x]);
        }
    }
}

struct PartArgs {
    BatchView bv;
    const void *S;
    const float *gamma;
    const double *gamma64;
    float *lambda;
    double *lambda64, *ws;
    int max_iter, exit_mode, log_stride, warm;
    float tol;
    uint32_t *out_iters, *pcg_log;
};

// The instance of this CTA.  Read again by each phase instead of kept in registers across the elimination,
// which needs them (the opaque read of the CTA index keeps the compiler from holding on to it).
template <int FMT, class CF>
struct PartCtx {
    using ST = typename PartRows<FMT>::ST;
    static constexpr ptrdiff_t ks = FMT == 2 ? PK64 : PK;
    const PartArgs &A;
    int inst, n;
    ptrdiff_t kg0;
    __device__ __forceinline__ explicit PartCtx(const PartArgs &args) : A(args)
    {
        int cta;
        asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(cta));
        inst = A.bv.b0 + cta / CF::CL;
        n = A.bv.N(inst);
        kg0 = A.bv.off(inst);
    }
    __device__ __forceinline__ const ST *rows() const { return reinterpret_cast<const ST *>(A.S) + ks * kg0; }
    __device__ __forceinline__ double *work() const { return A.ws + kg0 * QW_STRIDE; }
    __device__ __forceinline__ double &vec(int slot, int e) const
    {
        return A.ws[(kg0 + e / NS) * QW_STRIDE + slot + e % NS];
    }
    __device__ __forceinline__ double gam(int e) const
    {
        return FMT == 2 ? A.gamma64[NS * kg0 + e] : (double)A.gamma[NS * kg0 + e];
    }
};

// This lane's part of a lower bound of ||gamma - S lambda||^2 for the caller's lambda, by warp w of nw: the residual of one
// knot (lane pair c its row c), and a NaN if an entry of lambda is not finite.
// (Out of line: it would cost the elimination registers.)
template <int FMT, class CF>
__device__ __noinline__ double part_start_bound(const PartArgs &A, int w, int nw)
{
    using ST = typename PartRows<FMT>::ST;
    constexpr ptrdiff_t ks = PartCtx<FMT, CF>::ks;
    extern __shared__ __align__(16) double part_dyn_smem[];
    const int *lay = PartSmem<CF>(part_dyn_smem).lay;
    const PartCtx<FMT, CF> cx(A);
    const int lo = lay[3], hi = lay[4];
    const int lane = threadIdx.x & 31, c = lane >> 1, h = lane & 1, cl = c < NS ? c : NS - 1;
    const float *lam = cx.A.lambda + NS * cx.kg0;
    double s = 0.0;
#pragma unroll 8
    for (int e = NS * lo + 32 * w + lane; e < NS * hi; e += 32 * nw) s = fma(0.0, (double)lam[e], s);
    const int k = lo + (hi - lo) * w / nw;
    if (k >= hi) return s;
    const bool left = k > 0, right = k < cx.n - 1;
    const ST *row = cx.rows() + ks * k;
    const float *x = lam + NS * k + h;
    double a = 0.0, b = 0.0, d = 0.0;
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        const int j = 2 * q + h;
        if (left) a = fma((double)row[cl + NS * j], (double)x[2 * q - NS], a);
        b = fma((double)row[PK_LEFT_N + tri_idx(cl, j)], (double)x[2 * q], b);
        if (right) d = fma((double)row[ks + j + NS * cl], (double)x[2 * q + NS], d);
    }
    a += b + d;
    const double r = cx.gam(NS * k + cl) - (a + __shfl_xor_sync(0xffffffffu, a, 1));
    return h == 0 && c < NS ? fma(r, r, s) : s;
}

// y in xv -> x of M x = y in xv, and S x in the workspace (QW_SX); CHECK and first: bound as of part_start_bound, by the
// warps that wait for the separators
template <int FMT, class CF, bool CHECK>
__device__ __forceinline__ void part_apply(const PartArgs &A, bool first, double &bound)
{
    using ST = typename PartRows<FMT>::ST;
    constexpr int NW = CF::NW;
    constexpr ptrdiff_t ks = PartCtx<FMT, CF>::ks;
    extern __shared__ __align__(16) double part_dyn_smem[];
    const PartSmem<CF> ps(part_dyn_smem);
    const PartCtx<FMT, CF> cx(A);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = part_rank<CF>(), part = rank * CF::WC + warp;
    const int c = lane >> 1, h = lane & 1, cl = c < NS ? c : NS - 1;
    const int n = cx.n;
    part_sync<CF>();
    const int P = ps.lay[0], len0 = ps.lay[1], step = ps.lay[2];  // separators at len0 + j step
    auto sep_of = [&](int j) { return len0 + j * step; };
    const bool mid = part > 0 && part < P - 1, top = part < P - 1 || P == 1;
    const int pa = part == 0 ? 0 : sep_of(part - 1) + 1, pb = part >= P - 1 ? n - 1 : sep_of(part) - 1;
    double *xv = ps.xv, *scw = ps.buf + warp * QBUF;
    if (part < P) {
        if (mid) walk_part<FMT, CF, true>(cx.rows(), cx.work(), pa, pb, true, true);
        else walk_part<FMT, CF, false>(cx.rows(), cx.work(), pa, pb, top, P > 1);
    }
    part_sync<CF>();
    // ---- the separators' system, by two warps of CTA 0: from both ends toward the middle separator sm and back (one
    // warp's chain over all of them is twice as long: seven took 20 k cycles)
    if (rank == 0 && warp < 2 && P >= 2) {
        const int sm = (P - 1) >> 1;  // of P - 1 separators
        const bool down = warp == 0;
        const int dj = down ? 1 : -1, js = down ? 0 : P - 2, cnt = down ? sm : P - 2 - sm;
        double a[7], e[7], b[7];
        auto rinv = [&](int j) { return ps.wmid + j * QINV; };
        auto region = [&](int p) { return part_peer<CF>(ps.stg + (p % CF::WC) * CF::REGION, p / CF::WC); };
        auto sep = [&](int j, double (&v)[7]) {
            const double *l = region(j) + lane, *r = region(j + 1) + (j + 1 < P - 1 ? QSEP : 0) + lane;
#pragma unroll
            for (int q = 0; q < 7; ++q) v[q] = l[32 * q] + r[32 * q];
        };
        // row i, column k of M_{s_{j+1}, s_j} at 32 (i >> 1) + 2 k + (i & 1)
        auto cpl = [&](int j) { return region(j + 1) + 2 * QSEP; };
        // E^T of separator j toward the middle: M_{s_{j+1}, s_j}^T, or M_{s_j, s_{j-1}}
        auto coup = [&](int j, double (&v)[7]) {
            const double *E = down ? cpl(j) + 32 * (cl >> 1) + (cl & 1) + 2 * h : cpl(j - 1) + 2 * cl + h;
#pragma unroll
            for (int q = 0; q < 7; ++q) v[q] = E[(down ? 4 : 32) * q];
        };
        auto keep = [&](int j) {
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                if (c <= 2 * q + h && c < NS) rinv(j)[2 * q * (q + 1) + lane] = a[q];
                if (c == NS) xv[NS * sep_of(j) + 2 * q + h] = e[q];
            }
        };
        if (cnt > 0) {
            double en[7], bn[7];
            sep(js, b);
            coup(js, en);
            for (int i = 0; i < cnt; ++i) {
                const int j = js + dj * i;
                if (down || i + 1 < cnt) {
                    sep(j + dj, bn);
                } else {
#pragma unroll
                    for (int q = 0; q < 7; ++q) bn[q] = 0.0;  // the middle one: its block is warp 0's
                }
#pragma unroll
                for (int q = 0; q < 7; ++q) {
                    a[q] = b[q];
                    e[q] = c < NS ? en[q] : b[q];
                    b[q] = bn[q];
                }
                if (i + 1 < cnt) coup(j + dj, en);
                part_step(a, e, b, scw, lane);
                keep(j);
            }
        } else if (down) {
            sep(sm, b);
        }
        double *upd = ps.wmid + CF::SEP_B + lane;
        PartBack pk;
        if constexpr (NW > 2) {
            if (!down) {
#pragma unroll
                for (int q = 0; q < 7; ++q) upd[32 * q] = cnt > 0 ? b[q] : 0.0;
            }
            asm volatile("bar.sync 1, 64;" ::: "memory");
        }
        if (down) {
            double zero[7];
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                if constexpr (NW > 2) b[q] += upd[32 * q];
                a[q] = b[q];
                e[q] = c < NS ? 0.0 : b[q];
                zero[q] = 0.0;
            }
            part_step(a, e, zero, scw, lane);
            keep(sm);
            __syncwarp();
            pk.load(rinv(sm), lane);
            pk.step(0.0, xv + NS * sep_of(sm), scw, lane);
        }
        if constexpr (NW > 2) asm volatile("bar.sync 1, 64;" ::: "memory");
        for (int i = cnt - 1; i >= 0; --i) {  // x_j from its neighbour toward the middle
            const int j = js + dj * i;
            const double *E = down ? cpl(j) + 2 * cl + h : cpl(j - 1) + 32 * (cl >> 1) + (cl & 1) + 2 * h;
            const double *xh = xv + NS * sep_of(j + dj) + h;
            double t = 0.0;  // -E^T x
#pragma unroll
            for (int q = 0; q < 7; ++q) t = fma(-E[(down ? 32 : 4) * q], xh[2 * q], t);
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            pk.load(rinv(j), lane);
            pk.step(t, xv + NS * sep_of(j), scw, lane);
        }
        if constexpr (CF::CL > 1) {  // to the other CTAs
            const int j0 = down ? 0 : sm + 1, nj = down ? sm + 1 : cnt;
            __syncwarp();
            for (int i = lane; i < NS * nj; i += 32) {
                const int e0 = NS * sep_of(j0 + i / NS) + i % NS;
                const double x = xv[e0];
#pragma unroll
                for (int r = 1; r < CF::CL; ++r) part_peer<CF>(xv, r)[e0] = x;
            }
        }
    }
    if (CHECK && first) {
        const int w0 = rank == 0 && P >= 2 ? (NW == 2 ? 1 : 2) : 0;
        if (warp >= w0) bound = part_start_bound<FMT, CF>(A, warp - w0, CF::WC - w0);
    }
    part_sync<CF>();
    // ---- backward through every part, and S x with it: a staged step is L^{-1} of the knot it solves and a row
    // of S.  Top-down parts go through the rows r = right separator .. pa: t = L_r^T x_r, then x_{r-1}, then row r
    // of S x; the last part through the rows r = pa .. pb: t = L_r x_{r-1}, then x_r, then row r - 1 of S x.
    // L_pa^T x_pa belongs to the left separator's row (sacc).
    double *sacc = ps.wmid + CF::SEP_SX;
    double *sleft = part > 0 ? part_peer<CF>(sacc, (part - 1) / CF::WC) + NS * ((part - 1) % CF::WC) : sacc;
    if (part < P) {
        double *stg = ps.stg + warp * CF::REGION;
        const ST *Sb = cx.rows();
        double *wsb = cx.work();
        const int len = pb >= pa ? pb - pa + 1 : 0, r0 = top ? (P > 1 ? pb + 1 : pb) : pa;
        const int count = top ? r0 - pa + 1 : len;
        auto stage = [&](int i) {
            if (i < count) {
                double *sl = stg + (i % CF::SB) * QBACK_D;
                const int r = top ? r0 - i : r0 + i, k = top ? r - 1 : r;
                if (k >= pa) warp_stage<QINV / 2>(sl, wsb + (ptrdiff_t)k * QW_STRIDE, lane);
                warp_stage<PartRows<FMT>::ROW_CHUNKS>(sl + QINV, Sb + ks * r, lane);
            }
            cp_async_commit();
        };
        int tri[7];
#pragma unroll
        for (int q = 0; q < 7; ++q) tri[q] = PK_LEFT_N + tri_idx(cl, 2 * q + h);
        double fr[7];
        auto ld_f = [&](int k) {
            const double *p = wsb + (ptrdiff_t)k * QW_STRIDE + QW_F + NS * cl + h;
#pragma unroll
            for (int q = 0; q < 7; ++q) fr[q] = p[2 * q];
        };
        auto dot = [&](const ST *M, int stride, const double (&x)[7]) {
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for (int q = 0; q < 7; ++q) (q & 1 ? s1 : s0) = fma((double)M[stride * q], x[q], q & 1 ? s1 : s0);
            return s0 + s1;
        };
        auto dot_diag = [&](const ST *M, const double (&x)[7]) {
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for (int q = 0; q < 7; ++q) (q & 1 ? s1 : s0) = fma((double)M[tri[q]], x[q], q & 1 ? s1 : s0);
            return s0 + s1;
        };
        auto pair = [](double v) { return v + __shfl_xor_sync(0xffffffffu, v, 1); };
        const double *xs = xv + NS * (mid ? pa - 1 : 0) + h;
        const int lc = NS * cl + h, lr = cl + NS * h;  // column (row) cl of a left block: strides 2 (2 NS)
        const bool wr = h == 0 && c < NS;
        PartBack pk;
        double xr[7];
        auto ld_x = [&](int k) {
#pragma unroll
            for (int q = 0; q < 7; ++q) xr[q] = xv[NS * k + 2 * q + h];
        };
        if (top && P == 1) {  // one part and no separator: its last knot first
            pk.load(wsb + (ptrdiff_t)pb * QW_STRIDE, lane);
            pk.step(0.0, xv + NS * pb, scw, lane);
        }
        for (int i = 0; i < CF::SB - 1; ++i) stage(i);
        if (mid && len > 0) ld_f(pb);
        if (count > 0) ld_x(top ? r0 : pa - 1);
        double carry = 0.0;
        for (int i = 0; i < count; ++i) {
            __syncwarp();
            stage(i + CF::SB - 1);
            cp_async_wait<CF::SB - 1>();  // step i has landed
            __syncwarp();
            const double *sl = stg + (i % CF::SB) * QBACK_D;
            const ST *M = reinterpret_cast<const ST *>(sl + QINV);
            if (top) {
                const int r = r0 - i, k = r - 1;
                const double t = pair(dot(M + lc, 2, xr));  // L_r^T x_r
                double v = dot_diag(M, xr);
                if (k >= pa) {
                    pk.load(sl, lane);
                    double tf = 0.0;
                    if (mid) {
#pragma unroll
                        for (int q = 0; q < 7; ++q) tf = fma(-fr[q], xs[2 * q], tf);
                        tf = pair(tf);
                        if (k > pa) ld_f(k - 1);
                    }
                    pk.step(t + tf, xv + NS * k, scw, lane);
                } else if (part > 0 && wr) {
                    sleft[c] = t;
                }
                if (r > 0) {
                    ld_x(k);
                    v += dot(M + lr, 2 * NS, xr);
                }
                v = pair(v) + carry;
                if (wr) wsb[(ptrdiff_t)r * QW_STRIDE + QW_SX + c] = v;
                carry = t;
            } else {
                const int r = r0 + i;
                const double t = pair(dot(M + lr, 2 * NS, xr));  // L_r x_{r-1}
                pk.load(sl, lane);
                pk.step(t, xv + NS * r, scw, lane);
                ld_x(r);
                const double u = pair(dot(M + lc, 2, xr)), v = pair(dot_diag(M, xr));
                if (wr) {
                    if (i == 0) sleft[c] = u;
                    else wsb[(ptrdiff_t)(r - 1) * QW_STRIDE + QW_SX + c] = carry + u;
                }
                carry = t + v;
            }
        }
        cp_async_wait<0>();
        if (!top && wr) {
            if (count > 0) wsb[(ptrdiff_t)pb * QW_STRIDE + QW_SX + c] = carry;
            else sleft[c] = 0.0;
        }
    }
    part_sync<CF>();
    if (part < P - 1 && lane < NS) cx.work()[(ptrdiff_t)sep_of(part) * QW_STRIDE + QW_SX + lane] += sacc[NS * warp + lane];
    __syncthreads();
}

// sums of v[0 .. CNT-1] over the instance's threads, in a fixed order (set: alternate between calls)
template <class CF, int CNT, int LEN>
__device__ __forceinline__ void part_sum(double (&v)[LEN], int set)
{
    static_assert(CNT <= LEN && CNT <= RED_N + 1, "the reduction's slots");
    extern __shared__ __align__(16) double part_dyn_smem[];
    double *all = PartSmem<CF>(part_dyn_smem).red, *red = all + set * CF::NW * RED_N;
    double *more = all + (2 * RED_N + set) * CF::NW;
    const int lane = threadIdx.x & 31, part = part_rank<CF>() * CF::WC + (threadIdx.x >> 5);
#pragma unroll
    for (int q = 0; q < CNT; ++q) {
        const double s = warp_sum(v[q]);
        if (lane < CF::CL) *part_peer<CF>(q < RED_N ? red + RED_N * part + q : more + part, lane) = s;
    }
    part_sync<CF>();
#pragma unroll
    for (int q = 0; q < CNT; ++q) {
        double s = 0.0;
        for (int w = 0; w < CF::NW; ++w) s += q < RED_N ? red[RED_N * w + q] : more[w];
        v[q] = s;
    }
}

// the vector entries of this CTA's knots, from this thread's first one on (every 32 WC-th is its own)
template <class CF>
struct PartRange {
    int first, end;
    __device__ __forceinline__ PartRange()
    {
        extern __shared__ __align__(16) double part_dyn_smem[];
        const int *lay = PartSmem<CF>(part_dyn_smem).lay;
        first = NS * lay[3] + threadIdx.x;
        end = NS * lay[4];
    }
};

// r = gamma - S lambda (the workspace's lambda; given: the caller's, copied there first) into the workspace and r . r; a
// rare path
template <int FMT, class CF>
__device__ __noinline__ double part_true_residual(const PartArgs &A, int set, bool given = false)
{
    const PartCtx<FMT, CF> cx(A);
    if (given) {
        const PartRange<CF> rg;
        for (int e = rg.first; e < rg.end; e += 32 * CF::WC) cx.vec(QW_LAM, e) = (double)A.lambda[NS * cx.kg0 + e];
    }
    const typename PartRows<FMT>::ST *Sb = cx.rows();
    constexpr ptrdiff_t ks = PartCtx<FMT, CF>::ks;
    double s[1] = {0.0};
    part_sync<CF>();
    const PartRange<CF> rg;
    for (int e = rg.first; e < rg.end; e += 32 * CF::WC) {
        const int k = e / NS, i = e % NS;
        const typename PartRows<FMT>::ST *row = Sb + ks * k;
        double a = 0.0;
        for (int j = 0; j < NS; ++j) {
            if (k > 0) a = fma((double)row[i + NS * j], cx.vec(QW_LAM, e - i - NS + j), a);
            a = fma((double)row[PK_LEFT_N + tri_idx(i, j)], cx.vec(QW_LAM, e - i + j), a);
            if (k < cx.n - 1) a = fma((double)row[ks + j + NS * i], cx.vec(QW_LAM, e - i + NS + j), a);
        }
        const double r = cx.gam(e) - a;
        cx.vec(QW_RES, e) = r;
        s[0] = fma(r, r, s[0]);
    }
    part_sum<CF, 1>(s, set);
    return s[0];
}

// CHECK: a caller's lambda that meets the tolerance is the result.  Any other leads to the solution from 0 too, so whether it
// does is told by a part of its residual, formed by warps that wait for the separators, and by all of it only where that
// part does not exclude it: a residual ahead of the elimination took 3.6 us more a launch at 32 knots (27 us in all) and 62
// at 512 x 128 (186), the part takes 0 and 12.  (A kernel of its own: its code costs the one that starts from 0 nine us at
// 512 x 128.)  A.warm without CHECK iterates from the caller's lambda.
template <int FMT, class CF, bool CHECK>
__global__ void __launch_bounds__(32 * CF::WC, CF::MINB) pcg_part_kernel(const __grid_constant__ PartArgs A)
{
    static_assert(FMT == 1 || FMT == 2, "packed rows only");
    constexpr int NT = 32 * CF::WC;
    extern __shared__ __align__(16) double part_dyn_smem[];
    double *xv = PartSmem<CF>(part_dyn_smem).xv;
    const int tid = threadIdx.x;
    {
        const PartCtx<FMT, CF> cx(A);
        if (!A.bv.active(cx.inst)) return;  // (the whole cluster)
        int lo = 0, hi = cx.n;
        const PartLayout<CF::NW> L = part_layout<CF::NW>(cx.n, CF::EDGE);
        const int sep_step = CF::NW > 2 ? L.s[CF::NW > 2 ? 1 : 0] - L.s[0] : 0;
        if constexpr (CF::CL > 1) {  // the CTA's parts and their right separators
            const int f = part_rank<CF>() * CF::WC, l = f + CF::WC - 1;
            lo = f == 0 ? 0 : (f < L.P ? L.s[0] + (f - 1) * sep_step + 1 : cx.n);
            hi = l >= L.P - 1 ? cx.n : L.s[0] + l * sep_step + 1;
        }
        if (tid == 0) {
            int *lay = PartSmem<CF>(part_dyn_smem).lay;
            lay[0] = L.P;
            lay[1] = L.s[0];
            lay[2] = sep_step;
            lay[3] = lo;
            lay[4] = hi;
        }
        for (int e = NS * lo + tid; e < NS * hi; e += NT) xv[e] = cx.gam(e);
    }
    int it = 0, set = 0;
    bool conv = false, bad = false, in_xv = false;
    bool has_res = false;  // r and lambda are in the workspace (before: r = gamma, lambda = 0)
    double eta = 0.0, gg = 0.0, alpha = 0.0;
    if (A.warm) {
        part_sync<CF>();
        const PartCtx<FMT, CF> cx(A);
        const PartRange<CF> rg;
        double g2[2] = {0.0, 0.0};  // gamma . gamma; entries of lambda that are not 0
        for (int e = rg.first; e < rg.end; e += NT) {
            const double lam = (double)A.lambda[NS * cx.kg0 + e];
            cx.vec(QW_LAM, e) = lam;
            g2[0] = fma(xv[e], xv[e], g2[0]);
            g2[1] += lam != 0.0 ? 1.0 : 0.0;
        }
        part_sum<CF, 2>(g2, set);
        if (g2[1] > 0.0) {
            gg = g2[0];
            part_true_residual<FMT, CF>(A, set ^ 1);
            for (int e = rg.first; e < rg.end; e += NT) xv[e] = cx.vec(QW_RES, e);
            has_res = true;
        } else {
            set ^= 1;
        }
    }
    auto converged = [&](double e, double r2) {
        return A.exit_mode == 0 ? (r2 <= (double)A.tol * (double)A.tol * gg) : (fabs(e) < (double)A.tol);
    };
    for (;;) {
        double bound = 0.0;
        part_apply<FMT, CF, CHECK>(A, it == 0, bound);
        const PartCtx<FMT, CF> cx(A);
        const PartRange<CF> rg;
        double dd[4] = {0.0, 0.0, 0.0, bound};  // r . z, r . r with z = -x; x . S x; the start's bound
        // the thread's first KEEP entries of r and S x stay in registers for the new residual's norm
        constexpr int KEEP = 8;
        double rk[KEEP], sk[KEEP];
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const int e = rg.first + NT * i;
            rk[i] = sk[i] = 0.0;
            if (e < rg.end) {
                rk[i] = has_res ? cx.vec(QW_RES, e) : cx.gam(e);
                sk[i] = cx.vec(QW_SX, e);
            }
        }
        auto dots = [&](double r, double x, double sx) {
            dd[0] = fma(-x, r, dd[0]);
            dd[1] = fma(r, r, dd[1]);
            dd[2] = fma(x, sx, dd[2]);
        };
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if (rg.first + NT * i < rg.end) dots(rk[i], xv[rg.first + NT * i], sk[i]);
        for (int e = rg.first + NT * KEEP; e < rg.end; e += NT)
            dots(has_res ? cx.vec(QW_RES, e) : cx.gam(e), xv[e], cx.vec(QW_SX, e));
        part_sum<CF, CHECK ? 4 : 3>(dd, set);
        set ^= 1;
        if (it == 0) {
            if (!has_res) gg = dd[1];
            conv = CHECK ? gg == 0.0 : converged(dd[0], dd[1]);
            if (CHECK && !conv && !(dd[3] > (double)A.tol * (double)A.tol * gg)) {
                const double r0 = part_true_residual<FMT, CF>(A, set, true);
                set ^= 1;
                bad = !isfinite(r0);
                conv = converged(0.0, r0);
                if (bad || conv) {
                    has_res = true;  // the start is the result
                    break;
                }
            }
        } else {
            if (!isfinite(dd[0])) {
                bad = true;
                break;
            }
            if (A.exit_mode != 0) conv = converged(dd[0], dd[1]);
        }
        if (conv || it >= A.max_iter) {
            eta = dd[0];
            break;
        }
        double psp = dd[2];  // p . S p, p = z on the first iteration
        if (it > 0) {        // p = z + beta p, S p = S z + beta S p
            const double beta = dd[0] / eta;
            double d1[1] = {0.0};
            for (int e = rg.first; e < rg.end; e += NT) {
                const double p = fma(beta, cx.vec(QW_P, e), -xv[e]), v = fma(beta, cx.vec(QW_V, e), -cx.vec(QW_SX, e));
                xv[e] = -p;
                cx.vec(QW_SX, e) = -v;
                d1[0] = fma(p, v, d1[0]);
            }
#pragma unroll
            for (int i = 0; i < KEEP; ++i)
                if (rg.first + NT * i < rg.end) sk[i] = cx.vec(QW_SX, rg.first + NT * i);
            part_sum<CF, 1>(d1, set);
            set ^= 1;
            psp = d1[0];
        }
        eta = dd[0];
        alpha = eta / psp;  // from here on xv = -p, QW_SX = -S p
        if (!isfinite(alpha)) {
            bad = true;
            break;
        }
        double r2[1] = {0.0};
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const double rn = fma(alpha, sk[i], rk[i]);
            r2[0] = fma(rn, rn, r2[0]);
        }
        for (int e = rg.first + NT * KEEP; e < rg.end; e += NT) {
            const double rn = fma(alpha, cx.vec(QW_SX, e), has_res ? cx.vec(QW_RES, e) : cx.gam(e));
            r2[0] = fma(rn, rn, r2[0]);
        }
        part_sum<CF, 1>(r2, set);
        set ^= 1;
        ++it;
        if (!has_res && A.exit_mode == 0 && converged(0.0, r2[0])) {
            conv = in_xv = true;  // lambda = alpha p
            break;
        }
        for (int e = rg.first; e < rg.end; e += NT) {
            cx.vec(QW_RES, e) = fma(alpha, cx.vec(QW_SX, e), has_res ? cx.vec(QW_RES, e) : cx.gam(e));
            cx.vec(QW_LAM, e) = fma(-alpha, xv[e], has_res ? cx.vec(QW_LAM, e) : 0.0);
            cx.vec(QW_P, e) = -xv[e];
            cx.vec(QW_V, e) = -cx.vec(QW_SX, e);
        }
        has_res = true;
        bool replaced = false;
        if (it % RR_PERIOD == 0) {
            r2[0] = part_true_residual<FMT, CF>(A, set);
            set ^= 1;
            replaced = true;
        }
        if (A.exit_mode == 0) {
            if (!isfinite(r2[0])) {
                bad = true;
                break;
            }
            if (converged(0.0, r2[0]) && !replaced && it > 1) {
                r2[0] = part_true_residual<FMT, CF>(A, set);
                set ^= 1;
            }
            if (converged(0.0, r2[0])) {
                conv = true;
                break;
            }
        }
        for (int e = rg.first; e < rg.end; e += NT) xv[e] = cx.vec(QW_RES, e);
    }
    const PartCtx<FMT, CF> cx(A);
    const PartRange<CF> rg;
    for (int e = rg.first; e < rg.end; e += NT) {
        // CHECK: a system that is not finite leaves the start
        const double none = CHECK && bad ? (double)A.lambda[NS * cx.kg0 + e] : 0.0;
        const double lam = in_xv ? -alpha * xv[e] : (has_res ? cx.vec(QW_LAM, e) : none);
        A.lambda[NS * cx.kg0 + e] = (float)lam;
        if (A.lambda64) A.lambda64[NS * cx.kg0 + e] = lam;
    }
    if (tid == 0 && part_rank<CF>() == 0) {
        const int inst = cx.inst;
        const uint32_t maxit = conv ? 0u : 1u;
        if (A.out_iters) {
            A.out_iters[2 * inst] = (uint32_t)it;
            A.out_iters[2 * inst + 1] = maxit | (bad ? 2u : 0u);
        }
        if (A.bv.st) {
            InstState &s = A.bv.st[inst];
            s.last_pcg_iters = it;
            s.last_pcg_exit = maxit;
            s.pcg_iters_total += it;
            s.pcg_maxiter_count += maxit;
            if (bad) s.exit_flags |= 4u;
            if (A.pcg_log && s.sqp_iters < (uint32_t)A.log_stride)
                A.pcg_log[(size_t)inst * A.log_stride + s.sqp_iters] = (uint32_t)it | (maxit << 31);
        }
    }
}

template <int FMT, class CF, bool CHECK>
static cudaError_t launch_part_t(const PartArgs &A, int max_n, cudaStream_t s)
{
    auto kern = pcg_part_kernel<FMT, CF, CHECK>;
    const size_t smem = CF::smem_bytes(max_n);
    const cudaError_t e = ensure_func_attrs((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = A.bv.B * CF::CL;
    cfg.blockDim = 32 * CF::WC;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = CF::CL;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = CF::CL > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, A);
}

// The variants: every warp of them has 255 registers (at 128, which four 4-warp CTAs per SM need, the
// elimination's loads serialise: 1.8 k -> 2.8 k cycles per edge step of a lone warp), so eight warps share an SM.
// Staging slots: the few-instance variants prefetch deeper, their sweeps being bound by the latency of L2.
using Part32 = PartCfg<8, 4, 6, 1, 15>;
using Part16 = PartCfg<4, 4, 6, 1, 15>;
using Part8x2 = PartCfg<2, 4, 6, 1, 15>;
using Part8 = PartCfg<1, 8, 6, 1, 15>;
using Part4 = PartCfg<1, QUAD_NWARP, 4, 2, QUAD_EDGE>;
using Part2 = PartCfg<1, 2, 3, 4, 13>;

// The variant of a batch.  More parts shorten an instance's chain but add the middle parts' work (about 1.6 of an edge
// part's per knot) and a separator each to the two-sided chain (3.3 k cycles for two of them); a cluster spreads the parts
// over SMs that would be idle, one warp per scheduler (2.4 k cycles per edge step against 3.3 k at two), and costs about
// 1.3 k cycles per cluster barrier.  Measured, us per launch (1 CTA of 4 / 1 of 8 / 2 x 4 / 4 x 4 / 8 x 4 warps), one instance:
// n = 16 20 / 20 / 29 / 24 / 25, n = 32 29 / 27 / 29 / 31 / 33, n = 48 40 / 37 / 35 / 36 / 41, n = 64 47 / 43 / 39 / 37 / 46,
// n = 128 85 / 72 / 60 / 47 / 52, n = 200 127 / 105 / 85 / 60 / 61, n = 300 185 / 149 / 117 / 76 / 72, n = 511 308 / 244 / 189
// / 113 / 85.  Clusters of 8 fit 14 or 15 times at once, of 4 33 times and of 2 74 times (n = 511, 16 instances: 166 us with
// 8 x 4, 114 with 4 x 4; n = 128, 35 instances: 62 with 4 x 4, 61 with 2 x 4; n = 64, 74 instances: 40 with 2 x 4, 46 with 8).
// Above one instance per SM 4 and 2 warps (us, 8 / 4 / 2 warps): n = 64, 200 instances 93 / 67 / 74, 400 instances
// 142 / 127 / 96.
int part_variant(int B, int max_n, int num_sms)
{
    if (B > num_sms) return B <= 2 * num_sms ? PART_4 : PART_2;
    if (max_n < 24) return PART_4;
    if (max_n < 48) return PART_8;
    if (max_n >= 256 && 12 * B <= num_sms) return PART_32;
    if (9 * B <= 2 * num_sms) return PART_16;
    return 2 * B <= num_sms ? PART_8X2 : PART_8;
}

template <class CF>
static cudaError_t launch_part_f(const PartArgs &A, int max_n, int fmt, bool check, cudaStream_t s)
{
    if (check) return fmt == 2 ? launch_part_t<2, CF, true>(A, max_n, s) : launch_part_t<1, CF, true>(A, max_n, s);
    return fmt == 2 ? launch_part_t<2, CF, false>(A, max_n, s) : launch_part_t<1, CF, false>(A, max_n, s);
}

cudaError_t launch_pcg_part(const BatchView &bv, int max_n, int fmt, const void *S, const float *gamma,
                            const double *gamma64, float *lambda, double *lambda64, double *ws, int max_iter,
                            float tol, int exit_mode, uint32_t *out_iters, uint32_t *pcg_log, int log_stride,
                            int num_sms, cudaStream_t s, bool warm)
{
    // the exit test on r . z, and no iteration at all, take the start as it is
    const bool check = warm && exit_mode == 0 && max_iter > 0;
    const PartArgs A{bv,       S,         gamma,      gamma64, lambda,    lambda64, ws,
                     max_iter, exit_mode, log_stride, warm && !check ? 1 : 0, tol, out_iters, pcg_log};
    switch (bv.part_variant ? bv.part_variant : part_variant(bv.B, max_n, num_sms)) {
    case PART_32: return launch_part_f<Part32>(A, max_n, fmt, check, s);
    case PART_16: return launch_part_f<Part16>(A, max_n, fmt, check, s);
    case PART_8X2: return launch_part_f<Part8x2>(A, max_n, fmt, check, s);
    case PART_8: return launch_part_f<Part8>(A, max_n, fmt, check, s);
    case PART_4: return launch_part_f<Part4>(A, max_n, fmt, check, s);
    default: return launch_part_f<Part2>(A, max_n, fmt, check, s);
    }
}

}  // namespace gpt

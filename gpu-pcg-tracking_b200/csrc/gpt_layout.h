// gpt_layout.h -- the part layout of the partitioned PCG (pcg_part_kernel): which knots each of
// the factoring warps owns and where the separator knots lie.  Plain C++ (host and device), so
// the CPU tests compile it and check the layout for every horizon.
#pragma once

#if defined(__CUDACC__)
#define GPT_HD __host__ __device__
#else
#define GPT_HD
#endif

namespace gpt {

// the variant of one CTA and four parts (Part4)
constexpr int QUAD_NWARP = 4, QUAD_EDGE = 15;

// NW: the most parts; edge: an edge part's length in tenths of a middle part's
template <int NW>
struct PartLayout {
    int P;
    int a[NW], b[NW];  // part p: knots a[p] .. b[p] (b[p] < a[p]: empty)
    int s[NW - 1];     // separator knots
};
template <int NW>
GPT_HD inline PartLayout<NW> part_layout(int n, int edge)
{
    PartLayout<NW> L;
    int P = NW;
    if (n < 2 * P) {
        P = (n + 1) / 2;
        P = P < 1 ? 1 : (P > NW ? NW : P);
    }
    L.P = P;
    const int nint = n - (P - 1);
    int len[NW] = {};
    if (P == 1) {
        len[0] = n;
    } else if (P == 2) {
        len[0] = nint / 2;
        len[1] = nint - len[0];
    } else {
        // the balanced length of a middle part rounded down, or up where that makes the longest walk shorter (a step of
        // a middle part takes edge tenths of an edge part's; sixteen parts of 128 knots: edges of 14 and 15 knots
        // beside middles of 6, or of 7 and 8 beside 7)
        int y = (10 * nint) / (2 * edge + 10 * (P - 2));
        int rest = nint - (P - 2) * y;
        const int up = rest - (P - 2), walk = edge * y > 5 * (rest + 1) ? edge * y : 5 * (rest + 1);
        if (up >= 0 && edge * (y + 1) < walk && 5 * (up + 1) < walk) {
            ++y;
            rest = up;
        }
        len[0] = rest / 2;
        for (int p = 1; p < P - 1; ++p) len[p] = y;
        len[P - 1] = rest - len[0];
    }
    int pos = 0;
    for (int p = 0; p < NW; ++p) {
        L.a[p] = pos;
        L.b[p] = pos + (p < P ? len[p] : 0) - 1;
        pos += p < P ? len[p] : 0;
        if (p < NW - 1) {
            L.s[p] = pos;
            if (p < P - 1) ++pos;
        }
    }
    return L;
}

using QuadLayout = PartLayout<QUAD_NWARP>;
GPT_HD inline QuadLayout quad_layout(int n) { return part_layout<QUAD_NWARP>(n, QUAD_EDGE); }

}  // namespace gpt

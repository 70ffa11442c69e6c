// clip_engine.cuh -- warp-cooperative exact clipping of tets against unit cells.
//
// The (tet, cell) pairs a CTA has listed are clipped by its warps, a lane per
// piece (a tet, 12 FP32 coordinates in the cell frame), in three kinds of
// steps, each with the same instructions on every lane:
//   * a build step turns 32 listed pairs into pieces, which go to the warp's
//     shared-memory pool, or to its last-face list if they cross one cell face;
//   * a split step takes up to 32 pieces from the pool (last in, first out)
//     and splits each by a cell face it crosses (of those, one with the fewest
//     of its vertices inside: next_face) into 1 or 3 inside pieces.  A child
//     outside a face is dropped; one inside all of them adds its 6x volume, as
//     exact 64-bit fixed point, to the accumulator of the pair it came from;
//     one that crosses a single face goes to the last-face list with its
//     volume; only the others go back to the pool;
//   * a last-face step sums the inside parts of up to 32 listed pieces: their
//     volumes times the inside fractions (from the edge parameters alone, no
//     cut points).
// A pair whose tet crosses several faces (up to 3^6 pieces) so spreads over
// the warp instead of serialising one lane.  What bounds it is issue, the ALU
// pipe (selects, flags) first.  One loop whose step did all of it, each lane
// in its own branch, had run ~640 instructions a step.  Octree leaves of a
// 192^3 lattice, the whole kernel, warp instructions and time: that loop
// 1.78e10, 25.4 ms; three kinds of steps, with selects free of branches
// (bit_sel), 1.43e10; flags as a byte per vertex 1.33e10, 17.7 ms; two FP32
// operations an instruction (fma2) 1.24e10, 17.1 ms; with the set-up's and
// the classification's share 1.20e10, 16.3 ms.
//
// The split keeps every piece positively oriented: the vertices are permuted
// (an even permutation) so that the k inside vertices come first, then the
// inside part is written as 1 tet (k = 1) or as a 3-tet prism decomposition
// (k = 2, 3) over the cut points on the crossing edges.
#pragma once

#include "geometry.cuh"

namespace adeco {

// inside-first even permutation (4 x 2 bits) and inside count per side mask
#define ADECO_SPLIT_PERM {228, 228, 177, 228, 210, 210, 201, 228, 99, 156, 135, 177, 78, 120, 54, 228}
#define ADECO_SPLIT_KIN {0, 1, 1, 2, 1, 2, 2, 3, 1, 2, 2, 3, 2, 3, 3, 4}
static const uint8_t h_split_perm[16] = ADECO_SPLIT_PERM;
static const int8_t h_split_kin[16] = ADECO_SPLIT_KIN;

// The tables are read with lane-dependent masks, which a constant-memory load
// serialises per distinct address; the entries are therefore taken from
// immediates (the permutation: a byte per mask, picked by a byte permute) and
// from the popcount (the inside count) -- the same values as
// ADECO_SPLIT_PERM / ADECO_SPLIT_KIN.
ADECO_HD inline int split_perm(int m)
{
#ifdef __CUDA_ARCH__
    const unsigned lo = __byte_perm(0xe4b1e4e4u, 0xe4c9d2d2u, m & 7), hi = __byte_perm(0xb1879c63u, 0xe436784eu, m & 7);
    return (int)(((m & 8) ? hi : lo) & 0xffu);
#else
    const unsigned long long w = (m & 8) ? 0xe436784eb1879c63ull : 0xe4c9d2d2e4b1e4e4ull;
    return (int)((w >> ((m & 7) * 8)) & 0xffu);
#endif
}
ADECO_HD inline int split_kin(int m)
{
#ifdef __CUDA_ARCH__
    return __popc((unsigned)m);
#else
    return __builtin_popcount((unsigned)m);
#endif
}

ADECO_HD inline float sel4(int i, float a, float b, float c, float d)
{
    return (i & 2) ? ((i & 1) ? d : c) : ((i & 1) ? b : a);
}
ADECO_HD inline float sel3(int i, float x, float y, float z) { return i == 0 ? x : (i == 1 ? y : z); }

// A select by a bit mask (all ones: a, zero: b), one logic instruction.  Where
// an expression selects among many candidates the compiler turns ternaries
// into branches (the cut of a piece: 33 branch instructions of 224, and most
// of its time); the mask form has none.
ADECO_HD inline unsigned bit_mask(bool c) { return c ? 0xffffffffu : 0u; }
ADECO_HD inline float bit_sel(unsigned m, float a, float b)
{
#ifdef __CUDA_ARCH__
    unsigned r;
    asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(r) : "r"(m), "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
    return __uint_as_float(r);
#else
    return m ? a : b;
#endif
}

// x limited to [0, 1]
ADECO_HD inline float sat01(float x)
{
#ifdef __CUDA_ARCH__
    return __saturatef(x);
#else
    return fminf(fmaxf(x, 0.f), 1.f);
#endif
}

// 6 inside bits of a point: bit 2a = (x_a > 0), bit 2a+1 = (x_a < 1).  On the
// device from the sign bits of 0 - x and x - 1 (exact signs; a zero result is
// +0, a NaN has sign 0), shifted in one by one: half on the FMA pipe, where
// six compares and selects all go to the ALU pipe, the busiest one.
ADECO_HD inline int face_bits(float x, float y, float z)
{
#ifdef __CUDA_ARCH__
    unsigned b = __float_as_uint(__fsub_rn(z, 1.f)) >> 31;
    b = __funnelshift_l(__float_as_uint(__fsub_rn(0.f, z)), b, 1);
    b = __funnelshift_l(__float_as_uint(__fsub_rn(y, 1.f)), b, 1);
    b = __funnelshift_l(__float_as_uint(__fsub_rn(0.f, y)), b, 1);
    b = __funnelshift_l(__float_as_uint(__fsub_rn(x, 1.f)), b, 1);
    return (int)__funnelshift_l(__float_as_uint(__fsub_rn(0.f, x)), b, 1);
#else
    return (int)(x > 0.f) | ((int)(x < 1.f) << 1) | ((int)(y > 0.f) << 2) | ((int)(y < 1.f) << 3) |
           ((int)(z > 0.f) << 4) | ((int)(z < 1.f) << 5);
#endif
}

// The cut of a piece by face f, its vertices permuted to A B C D, the k
// inside ones first by an even permutation (the orientation is kept): the cut
// points E0..E3 of the cut edges -- k=1: AB AC AD; k=2: AC AD BC BD; k=3: AD
// BD CD -- snapped onto the face.  A vertex has N values, its
// coordinates last; the others (N = 6: barycentric weights) are interpolated
// with the coordinates' edge parameter.
// E3 is made for k = 2 only (BD; the other cases do not use it).  da..dd: the
// vertices' coordinate along f's axis.
template <int N>
ADECO_HD inline void cut_points(const float *A, const float *B, const float *C, const float *D, float da, float db,
                                float dc, float dd, int k, int f, float E[4][N])
{
    const int axis = f >> 1;
    const float plane = (f & 1) ? 1.f : 0.f;
    const unsigned k1 = bit_mask(k == 1), k2 = bit_mask(k == 2), k3 = bit_mask(k == 3);
    const unsigned ax[3] = {bit_mask(axis == 0), bit_mask(axis == 1), bit_mask(axis == 2)};
    // the ends of edges 0 and 1, 2 and 3
    const auto ends = [&](float a, float b, float c, float d, float2 in[2], float2 out[2]) {
        in[0] = make_float2(a, bit_sel(k3, b, a));
        out[0] = make_float2(bit_sel(k1, b, bit_sel(k2, c, d)), bit_sel(k1, c, d));
        in[1] = make_float2(bit_sel(k1, a, bit_sel(k2, b, c)), b);
        out[1] = make_float2(bit_sel(k2, c, d), d);
    };
    // two edges at a time; |dout - din| > 0 on a crossing edge
    float2 din[2], dout[2], t[2];
    ends(da, db, dc, dd, din, dout);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        // t = (plane - din) / (dout - din) as (din - plane) times minus the reciprocal
#ifdef __CUDA_ARCH__
        const float2 d = sub2(dout[e], din[e]);
        const float2 r = make_float2(rcp_approx(-d.x), rcp_approx(-d.y));
        const float2 q = fma2(r, fma2(d, r, both(1.f)), r);
#else
        const float2 q = make_float2(rcp_nr(din[e].x - dout[e].x), rcp_nr(din[e].y - dout[e].y));
#endif
        const float2 num = add2(din[e], both(-plane));
        t[e] = make_float2(sat01(num.x * q.x), sat01(num.y * q.y));
    }
#pragma unroll
    for (int x = 0; x < N; ++x) {
        float2 in[2], out[2];
        ends(A[x], B[x], C[x], D[x], in, out);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float2 cut = fma2(t[e], sub2(out[e], in[e]), in[e]);
            if (x >= N - 3) {
                const unsigned m = ax[x < N - 3 ? 0 : x - (N - 3)];
                cut = make_float2(bit_sel(m, plane, cut.x), bit_sel(m, plane, cut.y));
            }
            E[2 * e][x] = cut.x;
            E[2 * e + 1][x] = cut.y;
        }
    }
}

// Inside part of a cut piece as 1 or 3 positively oriented pieces, child
// 0..2:
//   k = 1: (A, Xab, Xac, Xad)
//   k = 2: (A, B, Xbc, Xbd) (A, Xbc, Xac, Xbd) (A, Xac, Xad, Xbd)
//   k = 3: (A, B, C, Xcd)  (A, B, Xcd, Xbd) (A, Xbd, Xcd, Xad)
// child_vertex picks vertex 1..3 of a child (vertex 0 is A) among the values
// of B, C and the cut points: coordinates, or any other 32-bit words of them.
ADECO_HD inline float child_vertex(int child, int v, unsigned k1, unsigned k2, float B, float C, const float E[4])
{
    if (child == 0) return v == 1 ? bit_sel(k1, E[0], B)
                                  : (v == 2 ? bit_sel(k1, E[1], bit_sel(k2, E[2], C)) : bit_sel(k2, E[3], E[2]));
    if (child == 1) return v == 1 ? bit_sel(k2, E[2], B) : (v == 2 ? bit_sel(k2, E[0], E[2]) : bit_sel(k2, E[3], E[1]));
    return v == 1 ? bit_sel(k2, E[0], E[1]) : (v == 2 ? bit_sel(k2, E[1], E[2]) : bit_sel(k2, E[3], E[0]));
}

template <int N>
ADECO_HD inline void split_child(int child, unsigned k1, unsigned k2, const float *A, const float *B, const float *C,
                                 const float E[4][N], float *p)
{
#pragma unroll
    for (int x = 0; x < N; ++x) {
        const float e[4] = {E[0][x], E[1][x], E[2][x], E[3][x]};
        p[x] = A[x];
#pragma unroll
        for (int v = 1; v < 4; ++v) p[N * v + x] = child_vertex(child, v, k1, k2, B[x], C[x], e);
    }
}

// Fraction of piece p inside face f (mask = 4-bit inside flags, 0 < mask <
// 15), from the edge parameters alone.  On an edge from inside vertex i to
// outside vertex o the plane sits at t = (plane - x_i) / (x_o - x_i); with u =
// 1 - t taken as (x_o - plane) / (x_o - x_i) so both keep their relative
// precision, and with the vertices ordered A B C D (inside first):
//   k = 1: t_AB t_AC t_AD                          (the corner tet at A)
//   k = 2: t_BC t_BD + t_AC t_BD u_BC + t_AC t_AD u_BD   (the 3-tet prism)
//   k = 3: 1 - u_AD u_BD u_CD = t_AD + u_AD (t_BD + u_BD t_CD)
// Every term is non-negative, so the fraction carries a few ulps of relative
// error and the inside volume needs no cut points and no child volumes.
// The same fraction for any linear function over the tet: x0..x3 its values
// at the vertices, inside = the side of `plane` given by mask.
ADECO_HD inline float side_fraction(float x0, float x1, float x2, float x3, int mask, float plane)
{
    const int pm = split_perm(mask), k = split_kin(mask);
    const bool k1 = k == 1, k2 = k == 2, k3 = k == 3;
    const float a = sel4(pm & 3, x0, x1, x2, x3), b = sel4((pm >> 2) & 3, x0, x1, x2, x3);
    const float c = sel4((pm >> 4) & 3, x0, x1, x2, x3), d = sel4((pm >> 6) & 3, x0, x1, x2, x3);
    // edges as in cut_points: k=1: AB AC AD; k=2: AC AD BC BD; k=3: AD BD CD
    const float in[4] = {a, k3 ? b : a, k1 ? a : (k2 ? b : c), b};
    const float out[4] = {k1 ? b : (k2 ? c : d), k1 ? c : d, k2 ? c : d, d};
    float t[4], u[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        // an unbiased reciprocal (rcp_nr): an approximate one biases the
        // fractions of all pairs the same way and shows in the total mass
        const float r = rcp_nr(out[e] - in[e]);
        t[e] = sat01((plane - in[e]) * r);
        u[e] = sat01((out[e] - plane) * r);
    }
    // all three formulas and a select: a branch by k runs them one after the other anyway
    const float f1 = t[0] * t[1] * t[2];
    const float f2 = fmaf(t[2], t[3], t[0] * (t[3] * u[2] + t[1] * u[3]));
    const float f3 = fmaf(u[0], fmaf(u[1], t[2], t[1]), t[0]);
    return k1 ? f1 : (k2 ? f2 : f3);
}

// 6x volume of the unit cube's part where G(u) = G0 + n.u > 0 (G0 a
// double-float pair).  The cube is first reflected along every axis where
// n_i < 0 (the volume does not change), so that n >= 0 and G grows along
// every edge path from corner 0 to corner 7.  The corner values are then
// formed exactly (TwoSum) and rounded once, which keeps that order, and the
// cube is split into the 6 tets around the diagonal 0-7, each of 6x volume 1:
// tet (0, a, b, 7) for the paths a -> b in {1,2,4} -> {3,5,6}, with values
// g0 <= ga <= gb <= g7.  The part of a tet where G > 0 is then a suffix of its
// path, and its fraction comes from the parameters t = g_in / (g_in - g_out)
// and u = 1 - t = -g_out / (g_in - g_out) of its crossing edges:
//   only 7 inside (gb <= 0 < g7):  t_70 t_7a t_7b        (the corner tet)
//   7, b inside (ga <= 0 < gb):    t_b0 t_ba + t_70 t_ba u_b0 + t_70 t_7a u_ba   (the prism)
//   0 outside (g0 <= 0 < ga):      t_a0 + u_a0 (t_b0 + u_b0 t_70)
// -- non-negative terms only, the same instructions on every lane, and the 19
// edge reciprocals shared by the 6 tets.  A face function turns a value a
// few ulps off its exact one, so a plane passing close to a corner keeps its
// relative precision.
ADECO_HD inline float halfspace_cube_vol6(F2 G0, float nx, float ny, float nz)
{
    G0 = f2_add(G0, F2{fminf(nx, 0.f), 0.f});
    G0 = f2_add(G0, F2{fminf(ny, 0.f), 0.f});
    G0 = f2_add(G0, F2{fminf(nz, 0.f), 0.f});
    nx = fabsf(nx);
    ny = fabsf(ny);
    nz = fabsf(nz);
    const F2x2 e12 = f2x2_add({both(G0.hi), both(G0.lo)}, make_float2(nx, ny));
    const F2x2 e45 = f2x2_add({make_float2(G0.hi, e12.hi.x), make_float2(G0.lo, e12.lo.x)}, both(nz));
    const F2x2 e36 = f2x2_add(e12, make_float2(ny, nz));
    const F2 e7 = f2_add(F2{e36.hi.x, e36.lo.x}, F2{nz, 0.f});
    const float g0 = G0.hi + G0.lo, g7 = e7.hi;
    const float ga[3] = {e12.hi.x, e12.hi.y, e45.hi.x};   // a = 1, 2, 4
    const float gb[3] = {e36.hi.x, e45.hi.y, e36.hi.y};   // b = 3, 5, 6
    if (!(g7 > 0.f)) return 0.f;
    if (g0 > 0.f) return 6.f;
    const float r70 = rcp_nr(g7 - g0);
    const float t70 = g7 * r70;
    float ta0[3], ua0[3], t7a[3], tb0[3], ub0[3], t7b[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float2 gab = make_float2(ga[i], gb[i]);
        const float2 r0 = rcp_nr2(sub2(both(g0), gab)), r7 = rcp_nr2(sub2(gab, both(g7)));
        const float2 t0 = mul2(gab, r0), u0 = mul2(both(-g0), r0), t7 = mul2(both(g7), r7);
        ta0[i] = t0.x;
        tb0[i] = t0.y;
        ua0[i] = u0.x;
        ub0[i] = u0.y;
        t7a[i] = t7.x;
        t7b[i] = t7.y;
    }
    // tets (a, b) by index into ga / gb: (1,3) (1,5) (2,3) (2,6) (4,5) (4,6)
    const int ia[6] = {0, 0, 1, 1, 2, 2}, ib[6] = {0, 1, 0, 2, 1, 2};
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < 6; q += 2) {  // two tets of the same a
        const int i = ia[q], j = ib[q], k = ib[q + 1];
        const float2 g = make_float2(gb[j], gb[k]), tb = make_float2(tb0[j], tb0[k]), ub = make_float2(ub0[j], ub0[k]);
        const float2 rba = rcp_nr2(sub2(both(ga[i]), g));
        const float2 tba = mul2(g, rba), uba = mul2(both(-ga[i]), rba);
        const float2 k1 = mul2(both(t70 * t7a[i]), make_float2(t7b[j], t7b[k]));
        const float2 k2 = fma2(tb, tba, mul2(both(t70), fma2(tba, ub, mul2(both(t7a[i]), uba))));
        const float2 k3 = fma2(both(ua0[i]), fma2(ub, both(t70), tb), both(ta0[i]));
        v += (g.x <= 0.f) ? k1.x : ((ga[i] <= 0.f) ? k2.x : k3.x);
        v += (g.y <= 0.f) ? k1.y : ((ga[i] <= 0.f) ? k2.y : k3.y);
    }
    return v;
}

// 2x2 minor a d - b c
ADECO_HD inline F2 f2_minor(F2 a, F2 d, F2 b, F2 c)
{
    const F2 bc = f2_mul(b, c);
    return f2_add(f2_mul(a, d), {-bc.hi, -bc.lo});
}

// The cell face a piece is clipped by next, from its vertices' 6-bit inside
// flags b0..b3 and the faces already done (`done`, one bit per face):
// returns 0 if the piece lies beyond a remaining face (dropped), 1 if it lies
// inside all of them (finished), else 2 with `face` the crossed face that has
// the fewest of the piece's vertices inside, `mask` those vertices and `last`
// set when no other face is crossed.  Fewest inside first: a single inside
// vertex gives a single child, the corner tet at that vertex, which often
// clears the other faces; two or three give three children.  Serial model on
// lattice-like tets, steps per clipped pair with the lowest crossed face
// first / this order: 19.1 / 8.7 at cells half a tet wide, 8.5 / 5.2 at
// tet-sized cells, 4.2 / 3.1 at cells two tets wide.
ADECO_HD inline int next_face(int b0, int b1, int b2, int b3, int done, int &face, int &mask, bool &last)
{
    const int all_in = b0 & b1 & b2 & b3, any_in = b0 | b1 | b2 | b3;
    const int relevant = 63 & ~done;
    const int next = (~all_in) & relevant;  // crossed, or entirely outside
    // per crossed face 1..3 vertices inside: odd -> 1 or 3, `two` -> at least 2
    const int odd = b0 ^ b1 ^ b2 ^ b3;
    const int two = (b0 & b1) | (b2 & b3) | ((b0 | b1) & (b2 | b3));
    const int one_in = next & odd & ~two, two_in = next & ~odd;
    const int pick = (one_in ? one_in : (two_in ? two_in : next)) | (next ? 0 : 1);
#ifdef __CUDA_ARCH__
    face = 31 - __clz(pick & -pick);
#else
    face = __builtin_ctz(pick);
#endif
    mask = ((b0 >> face) & 1) | (((b1 >> face) & 1) << 1) | (((b2 >> face) & 1) << 2) | (((b3 >> face) & 1) << 3);
    last = (next & (next - 1)) == 0;
    return (~any_in & relevant) ? 0 : (next ? 2 : 1);
}

// ---------------------------------------------------- barycentric clipping
// Fraction of a tet's volume inside the unit cube, for tets too flat for the
// FP32 engine.  A flat tet's volume L^2 h, computed from FP32 coordinates as
// a determinant, carries an error ~ 2^-24 L^3 -- relative 2^-24 kappa.  Here
// every piece also carries its barycentric coordinates in the tet (4 weights
// per vertex): clipping is affine, so a cut point's weights follow from the
// same edge parameter t as its coordinates, and a piece's share of the tet is
// the determinant of its weights -- well conditioned whatever the tet's
// shape; the mass is that share times the tet's exact mass.  Face tests, cut
// points (snapped onto the face), splits, last-face fractions and the face
// order are the engine's, on the piece's own coordinates.

// A piece's signed share of the tet: the determinant of its weight
// differences (the weights of vertices 1..3 minus those of vertex 0), from
// exact differences in double-float.  A record carries a vertex's weights
// of tet vertices 1..3 only: the weight of vertex 0 (one minus their sum)
// does not enter the determinant.  Signed: every piece keeps the tet's
// orientation, and |det| would round near-degenerate pieces up and bias the
// sum.
ADECO_HD inline F2 bary_share(const float *w)
{
    F2 d[3][3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) d[j][i] = f2_two_sum(w[3 * (j + 1) + i], -w[i]);
    const F2 m0 = f2_minor(d[1][1], d[2][2], d[1][2], d[2][1]);
    const F2 m1 = f2_minor(d[1][0], d[2][2], d[1][2], d[2][0]);
    const F2 m2 = f2_minor(d[1][0], d[2][1], d[1][1], d[2][0]);
    const F2 t1 = f2_mul(d[0][1], m1);
    return f2_add(f2_add(f2_mul(d[0][0], m0), {-t1.hi, -t1.lo}), f2_mul(d[0][2], m2));
}

constexpr int kBaryRec = 24;  // a barycentric piece: 12 weights (3 per vertex), then 12 coordinates

// the tet itself: vertex v (1..3) has weight 1 for tet vertex v, vertex 0 none
ADECO_HD inline void bary_identity(float *r)
{
#pragma unroll
    for (int i = 0; i < 12; ++i) r[i] = (i & 3) == 3 ? 1.f : 0.f;  // entries 3, 7, 11
}

// The share inside the unit cube of one barycentric piece rec0 whose faces
// in done0 are already done, clipped serially with a stack, for checks on the
// host: faces, cut points, children and shares by the warp engine's functions
// (clip_bary_pairs).
inline F2 clip_bary_serial(const float *rec0, int done0)
{
    constexpr int kDepth = 16;
    float stk[kDepth][24];  // a vertex's 3 weights and 3 coordinates, as the engine's pool
    int sdone[kDepth];
    for (int q = 0; q < 4; ++q)
        for (int i = 0; i < 3; ++i) {
            stk[0][6 * q + i] = rec0[3 * q + i];
            stk[0][6 * q + 3 + i] = rec0[12 + 3 * q + i];
        }
    sdone[0] = done0;
    int sp = 1;
    F2 acc = {0.f, 0.f};
    while (sp > 0) {
        --sp;
        float V[4][6], w[12];
        int bits[4];
        for (int q = 0; q < 4; ++q) {
            for (int i = 0; i < 6; ++i) V[q][i] = stk[sp][6 * q + i];
            for (int i = 0; i < 3; ++i) w[3 * q + i] = V[q][i];
            bits[q] = face_bits(V[q][3], V[q][4], V[q][5]);
        }
        const int done = sdone[sp];
        int f = 0, mask = 0;
        bool last = false;
        const int code = next_face(bits[0], bits[1], bits[2], bits[3], done, f, mask, last);
        if (code == 0) continue;  // beyond a face
        if (code == 1) {
            acc = f2_add(acc, bary_share(w));
            continue;
        }
        const int ax = 3 + (f >> 1);
        if (last) {  // last crossed face: the inside fraction of the piece
            acc = f2_add(acc, f2_mul_f(bary_share(w), side_fraction(V[0][ax], V[1][ax], V[2][ax], V[3][ax], mask,
                                                                    (f & 1) ? 1.f : 0.f)));
            continue;
        }
        const int pm = split_perm(mask), k = split_kin(mask), n = k == 1 ? 1 : 3;
        if (sp + n > kDepth) continue;  // cannot happen: at most 2 pending pieces per face level
        const float *A = V[pm & 3], *B = V[(pm >> 2) & 3], *C = V[(pm >> 4) & 3], *D = V[(pm >> 6) & 3];
        float E[4][6];
        cut_points<6>(A, B, C, D, A[ax], B[ax], C[ax], D[ax], k, f, E);
        for (int c = 0; c < n; ++c) {
            split_child<6>(c, bit_mask(k == 1), bit_mask(k == 2), A, B, C, E, stk[sp]);
            sdone[sp] = done | (1 << f);
            ++sp;
        }
    }
    return acc;
}

constexpr int kVolShift = 56;  // fixed point of 6x piece volumes (each <= 6)
static_assert(kVolShift == 56, "vol_fixed scales by 0x1p56f");

ADECO_HD inline long long vol_fixed(float v6)
{
#ifdef __CUDA_ARCH__
    return __float2ll_rn(v6 * 0x1p56f);  // the signed form of to_fixed(|v6|, kVolShift)
#else
    const unsigned long long m = to_fixed(fabsf(v6), kVolShift);
    return v6 < 0.f ? -(long long)m : (long long)m;
#endif
}

ADECO_HD inline float piece_vol6(const float p[12])
{
    return vol6_fast<float>(p, p + 3, p + 6, p + 9);
}

// state of one piece whose faces in `done` are done (next_face): code 0 =
// dropped, 1 = finished, 2 = crossing `face` with inside mask `mask`
ADECO_HD inline int piece_step(const float p[12], int done, int &face, int &mask, bool &last)
{
    return next_face(face_bits(p[0], p[1], p[2]), face_bits(p[3], p[4], p[5]), face_bits(p[6], p[7], p[8]),
                     face_bits(p[9], p[10], p[11]), done, face, mask, last);
}

// 6x volume, in fixed point, of a piece that needs no further split: inside
// every remaining face, or the part inside the last crossed one (last).
ADECO_HD inline long long leaf_volume(const float p[12], bool last, int f, int mask)
{
    const int axis = f >> 1;
    float v = piece_vol6(p);
    if (last)
        v *= side_fraction(sel3(axis, p[0], p[1], p[2]), sel3(axis, p[3], p[4], p[5]), sel3(axis, p[6], p[7], p[8]),
                           sel3(axis, p[9], p[10], p[11]), mask, (f & 1) ? 1.f : 0.f);
    return vol_fixed(v);
}

// Serial clipping of one piece whose faces in `done0` are done (used when the
// warp pool is full): depth-first over the same splits and last-face fractions, so the
// fixed-point sum is the warp engine's.
#ifdef __CUDA_ARCH__
__device__ __noinline__
#else
inline
#endif
long long clip_piece_serial(const float p0[12], int done0)
{
    constexpr int kDepth = 16;  // 2 pending pieces per face level + 3
    float stk[kDepth][12];
    int sdone[kDepth];
#pragma unroll
    for (int x = 0; x < 12; ++x) stk[0][x] = p0[x];
    sdone[0] = done0;
    int sp = 1;
    long long acc = 0;
    while (sp > 0) {
        --sp;
        float p[12];
#pragma unroll
        for (int x = 0; x < 12; ++x) p[x] = stk[sp][x];
        int face = 0, mask = 0;
        bool last = false;
        const int code = piece_step(p, sdone[sp], face, mask, last);
        if (code == 0) continue;
        if (code == 1) {
            acc += leaf_volume(p, false, face, mask);
            continue;
        }
        if (last) {
            acc += leaf_volume(p, true, face, mask);
            continue;
        }
        const int pm = split_perm(mask), k = split_kin(mask);
        float V[4][3], E[4][3];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int x = 0; x < 3; ++x) V[q][x] = sel4((pm >> (2 * q)) & 3, p[x], p[3 + x], p[6 + x], p[9 + x]);
        const int ax = face >> 1;
        cut_points<3>(V[0], V[1], V[2], V[3], sel3(ax, V[0][0], V[0][1], V[0][2]), sel3(ax, V[1][0], V[1][1], V[1][2]),
                      sel3(ax, V[2][0], V[2][1], V[2][2]), sel3(ax, V[3][0], V[3][1], V[3][2]), k, face, E);
        const int n = k == 1 ? 1 : 3;
        if (sp + 3 > kDepth) continue;  // cannot happen (depth <= 2*5 + 3)
        const int d = sdone[sp] | (1 << face);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (c >= n) continue;
            split_child<3>(c, bit_mask(k == 1), bit_mask(k == 2), V[0], V[1], V[2], E, stk[sp]);
            sdone[sp] = d;
            ++sp;
        }
    }
    return acc;
}

#ifdef __CUDACC__
// The warp engines hold a piece's inside flags as a byte per vertex (6 bits
// each): what holds for all or any of the vertices comes from two steps over
// the word, a vertex order is one byte permutation, and so are the flags of a
// child, whose vertices are picked from two words by its case.
__device__ __forceinline__ unsigned pack_flags(int b0, int b1, int b2, int b3)
{
    return (unsigned)(b0 + 256 * b1) + 65536u * (unsigned)(b2 + 256 * b3);
}
// face_bits of two points
__device__ __forceinline__ void face_bits2(const float *p, const float *q, int &bp, int &bq)
{
    unsigned b = 0, c = 0;
#pragma unroll
    for (int a = 2; a >= 0; --a) {
        const float2 x = make_float2(p[a], q[a]), m1 = both(-1.f);
        const float2 up = add2(x, m1), lo = fma2(x, m1, both(0.f));
        b = __funnelshift_l(__float_as_uint(up.x), b, 1);
        b = __funnelshift_l(__float_as_uint(lo.x), b, 1);
        c = __funnelshift_l(__float_as_uint(up.y), c, 1);
        c = __funnelshift_l(__float_as_uint(lo.y), c, 1);
    }
    bp = (int)b;
    bq = (int)c;
}
__device__ __forceinline__ unsigned face_flags(const float *p0, const float *p1, const float *p2, const float *p3)
{
    int b0, b1, b2, b3;
    face_bits2(p0, p1, b0, b1);
    face_bits2(p2, p3, b2, b3);
    return pack_flags(b0, b1, b2, b3);
}
__device__ __forceinline__ int flags_all(unsigned m)  // in bits 0..5
{
    const unsigned a = m & (m >> 16);
    return (int)(a & (a >> 8));
}
__device__ __forceinline__ int flags_any(unsigned m)
{
    const unsigned o = m | (m >> 16);
    return (int)(o | (o >> 8));
}
// The vertices' flags of face f as a 4-bit mask: bits 0, 8, 16, 24 of m >> f
// moved to 28..31 (no two products of the multiplication meet below).
__device__ __forceinline__ int flags_mask(unsigned m, int f)
{
    return (int)((((m >> f) & 0x01010101u) * 0x10204080u) >> 28);
}
// next_face's choice for a piece of which the faces in `next` (not 0) are crossed
__device__ __forceinline__ int flags_face(unsigned m, int next)
{
    const unsigned a = m & (m >> 16), o = m | (m >> 16), x = m ^ (m >> 16);
    const int odd = (int)(x ^ (x >> 8));
    const int two = (int)(a | (a >> 8) | (o & (o >> 8)));
    const int one_in = next & odd & ~two, two_in = next & ~odd;
    const int pick = one_in ? one_in : (two_in ? two_in : next);
    return 31 - __clz(pick & -pick);
}
// child_vertex as byte selectors: bytes 0..2 are A B C, bytes 4..7 E0..E3
__device__ __forceinline__ unsigned child_bytes(int child, unsigned k1, unsigned k2)
{
    if (child == 0) return k1 ? 0x6540u : (k2 ? 0x7610u : 0x6210u);
    return child == 1 ? (k2 ? 0x7460u : 0x5610u) : (k2 ? 0x7540u : 0x4650u);
}

// Two CTAs of 8 warps fill an SM's shared memory.  Every list's end costs a
// drain with few lanes and a wait, so a longer list gains, until the pools,
// which fine grids fill, get too small: no-allocation 96^3 / octree leaves
// 256^3 / one zoom grid in ms with a list of 896 2.73 / 31.0 / 3.41, 1152 2.47 /
// 29.8 / 3.22, 1280 2.44 / 29.8 / 3.16, 1408 (pool 71) 2.43 / 29.9 / 3.53.
constexpr int kPool = 80;    // pieces per warp pool
constexpr int kLast = 84;    // pieces at their last crossed face per warp
constexpr int kPairs = 1280;  // partial pairs a CTA lists

static_assert(kPool >= 32 + 3 && kLast >= 32 + 3, "one split step fits a full pool and list");

struct WarpPool {
    float v[12][kPool];         // the pieces' coordinates, a row per coordinate: a lane's four vertices come in
                                // any order by their addresses (rows of a multiple of 32, free of bank
                                // conflicts, were no faster)
    uint32_t flags[kPool];      // the vertices' inside flags, a byte each
    uint16_t owner[kPool];      // the piece's pair
    float last[5][kLast];       // pieces at their last face: 6x volume, the vertices' coordinate along its axis
    uint32_t last_meta[kLast];  // inside mask | upper face << 4 | owner << 8
};

// The partial pairs a CTA has listed and their 6x volumes.
template <int kCap>
struct PairListOf {
    int n[2];     // pairs listed, and the first pair no warp has taken: a list's counters are cleared
    int next[2];  // while the one before it is clipped, so lists alternate between two sets
    uint32_t cell[kCap];  // the pair's cell (the caller's encoding)
    uint8_t tet[kCap];    //   and its tet
    uint32_t vlo[kCap], vhi[kCap];  // fixed point 2^kVolShift

    __device__ __forceinline__ long long volume(int j) const
    {
        return (long long)(((unsigned long long)vhi[j] << 32) | vlo[j]);
    }
    // 64-bit add as two 32-bit shared-memory additions, the carry taken from
    // the first one's result (a 64-bit shared-memory atomic is a
    // compare-and-swap loop, which lanes of the same pair repeat)
    __device__ __forceinline__ void add(int j, long long v)
    {
        const unsigned lo = (unsigned)v;
        const unsigned old = atomicAdd(&vlo[j], lo);
        atomicAdd(&vhi[j], (unsigned)((unsigned long long)v >> 32) + (unsigned)(old + lo < old));
    }
    __device__ __forceinline__ void set(int j, long long v)
    {
        vlo[j] = (uint32_t)v;
        vhi[j] = (uint32_t)((unsigned long long)v >> 32);
    }
};
using PairList = PairListOf<kPairs>;

__device__ __forceinline__ void put_last(WarpPool &pool, int slot, const float p[12], float v6, int f, int mask, int owner)
{
    const unsigned ax = bit_mask(f < 2), ay = bit_mask(f < 4);
    pool.last[0][slot] = v6;
#pragma unroll
    for (int q = 0; q < 4; ++q) pool.last[1 + q][slot] = bit_sel(ax, p[3 * q], bit_sel(ay, p[3 * q + 1], p[3 * q + 2]));
    pool.last_meta[slot] = (uint32_t)(mask | ((f & 1) << 4) | (owner << 8));
}

// Clip the CTA's np listed pairs (build(j, p) writes pair j's tet in cell
// coordinates); every warp takes pairs from the list, 32 at a time, until none
// is left.  A pair's pieces stay with the warp that took it: on return
// list.volume(j) of this warp's pairs are their 6x volumes.  Returns the 32s
// it took, a bit each.
template <typename Build>
__device__ __forceinline__ uint64_t clip_pairs(WarpPool &pool, PairList &list, int *next, int np, Build build,
                                               unsigned &fallbacks)
{
    static_assert(kPairs <= 64 * 32 && kPool >= 63 && kLast >= 63, "a build step has room for 32 pairs");
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1;
    int top = 0, nlast = 0;
    uint64_t taken = 0;
    bool more_pairs = np > 0;
    for (;;) {
        if (nlast >= 32 || (nlast && !top && !more_pairs)) {
            // the inside parts of up to 32 pieces at their last face
            const int n = min(nlast, 32), idx = nlast - 1 - lane;
            if (lane < n) {
                const uint32_t m = pool.last_meta[idx];
                const float frac = side_fraction(pool.last[1][idx], pool.last[2][idx], pool.last[3][idx],
                                                 pool.last[4][idx], m & 15, (m & 16) ? 1.f : 0.f);
                list.add((int)(m >> 8), vol_fixed(pool.last[0][idx] * frac));
            }
            nlast -= n;
            __syncwarp();
            continue;
        }
        if (top < 32 && more_pairs) {
            // build step
            int j = 0;
            if (lane == 0) j = atomicAdd(next, 32);
            j = __shfl_sync(0xffffffffu, j, 0);
            more_pairs = j + 32 < np;
            if (j >= np) continue;
            taken |= 1ull << (j >> 5);
            const int nb = min(32, np - j);
            j += lane;
            bool push = false, last = false;
            float p[12];
            uint32_t flags = 0;
            int f = 0, mask = 0;
            long long v = 0;
            if (lane < nb) {
                build(j, p);
                flags = face_flags(p, p + 3, p + 6, p + 9);
                const int next = 63 & ~flags_all(flags);  // crossed, or entirely outside
                if ((63 & ~flags_any(flags)) == 0) {
                    push = (next & (next - 1)) != 0;
                    last = next && !push;
                    if (last) {
                        f = 31 - __clz(next);
                        mask = flags_mask(flags, f);
                    }
                    if (next == 0) v = vol_fixed(piece_vol6(p));
                }
                list.set(j, v);
            }
            const unsigned pushing = __ballot_sync(0xffffffffu, push), lasts = __ballot_sync(0xffffffffu, last);
            if (push) {
                const int slot = top + __popc(pushing & lt);
#pragma unroll
                for (int x = 0; x < 12; ++x) pool.v[x][slot] = p[x];
                pool.flags[slot] = flags;
                pool.owner[slot] = (uint16_t)j;
            }
            if (last) put_last(pool, nlast + __popc(lasts & lt), p, piece_vol6(p), f, mask, j);
            top += __popc(pushing);
            nlast += __popc(lasts);
            __syncwarp();
            continue;
        }
        if (!top) return taken;
        // split step: lane l takes slot top - 1 - l
        const int n = min(top, 32), idx = top - 1 - lane;
        int owner = 0;
        int code[3] = {0, 0, 0};  // per child: 0 dropped, 1 inside, 2 at its last face, 3 to split further
        uint32_t cflags[3];
        int cnext[3];
        float A[3], B[3], C[3], E[4][3];
        unsigned k1 = 0, k2 = 0;
        if (lane < n) {
            // A done face has all four flags 0, which no other face of a pool
            // piece can have (the piece would lie outside it): no done set is kept.
            const uint32_t m = pool.flags[idx];
            owner = pool.owner[idx];
            const int left = 63 & flags_any(m);
            const int f = flags_face(m, left & ~flags_all(m)), mask = flags_mask(m, f);
            const int pm = split_perm(mask), k = split_kin(mask);
            const int ia = pm & 3, ib = (pm >> 2) & 3, ic = (pm >> 4) & 3, id = (pm >> 6) & 3;
            float D[3];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                A[x] = pool.v[3 * ia + x][idx];
                B[x] = pool.v[3 * ib + x][idx];
                C[x] = pool.v[3 * ic + x][idx];
                D[x] = pool.v[3 * id + x][idx];
            }
            const int ax = f >> 1;
            cut_points<3>(A, B, C, D, pool.v[3 * ia + ax][idx], pool.v[3 * ib + ax][idx], pool.v[3 * ic + ax][idx],
                          pool.v[3 * id + ax][idx], k, f, E);
            k1 = bit_mask(k == 1);
            k2 = bit_mask(k == 2);
            const int keep = left & ~(1 << f);
            const unsigned keep4 = 0x01010101u * (unsigned)keep;
            const unsigned wV = __byte_perm(m & keep4, 0, ia + 16 * ib + 256 * ic);  // bytes A B C
            const unsigned wE = face_flags(E[0], E[1], E[2], E[3]) & keep4;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                cflags[c] = __byte_perm(wV, wE, child_bytes(c, k1, k2));
                cnext[c] = keep & ~flags_all(cflags[c]);  // crossed, or entirely outside
                const bool out = (keep & ~flags_any(cflags[c])) != 0 || (c > 0 && k1);
                code[c] = out ? 0 : (cnext[c] == 0 ? 1 : ((cnext[c] & (cnext[c] - 1)) == 0 ? 2 : 3));
            }
        }
        unsigned sm[3], lm[3];  // the lanes whose child c goes to the pool / to the last-face list
        int ns = 0, nl = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sm[c] = __ballot_sync(0xffffffffu, code[c] == 3);
            lm[c] = __ballot_sync(0xffffffffu, code[c] == 2);
            ns += __popc(sm[c]);
            nl += __popc(lm[c]);
        }
        // When the children do not all fit, the first lanes for which they do
        // commit their step; the pieces of the others, the lower slots, stay
        // where they are.  Only when not even one step fits is a piece clipped
        // serially, with a local stack.
        int commit = n;
        if (top - n + ns > kPool || nlast + nl > kLast) {
            int s_incl = 0, l_incl = 0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                s_incl += __popc(sm[c] & (lt << 1 | 1));
                l_incl += __popc(lm[c] & (lt << 1 | 1));
            }
            const unsigned bad =
                __ballot_sync(0xffffffffu, lane < n && (top - (lane + 1) + s_incl > kPool || nlast + l_incl > kLast));
            if (bad) commit = __ffs(bad) - 1;
            const unsigned cm = commit < 32 ? (1u << commit) - 1 : 0xffffffffu;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sm[c] &= cm;
                lm[c] &= cm;
            }
            if (commit == 0) {
                if (lane == 0) {
                    float q[12];
#pragma unroll
                    for (int x = 0; x < 12; ++x) q[x] = pool.v[x][idx];
                    const uint32_t m = pool.flags[idx];
                    list.add(owner, clip_piece_serial(q, 63 & ~flags_any(m)));
                    ++fallbacks;
                }
                --top;
                __syncwarp();
                continue;
            }
        }
        top -= commit;
        __syncwarp();  // every lane has read its slot
        long long v = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (lane < commit && code[c]) {
                float ch[12];
                split_child<3>(c, k1, k2, A, B, C, E, ch);
                if (code[c] == 3) {
                    const int slot = top + __popc(sm[c] & lt);
#pragma unroll
                    for (int x = 0; x < 12; ++x) pool.v[x][slot] = ch[x];
                    pool.flags[slot] = cflags[c];
                    pool.owner[slot] = (uint16_t)owner;
                } else {
                    const float v6 = piece_vol6(ch);
                    if (code[c] == 1) {
                        v += vol_fixed(v6);
                    } else {
                        const int f = 31 - __clz(cnext[c]);
                        put_last(pool, nlast + __popc(lm[c] & lt), ch, v6, f, flags_mask(cflags[c], f), owner);
                    }
                }
            }
            top += __popc(sm[c]);
            nlast += __popc(lm[c]);
        }
        if (v) list.add(owner, v);
        __syncwarp();
    }
}

// ------------------------------------------- barycentric warp engine
// clip_pairs for pieces that carry barycentric weights: a vertex has 6 values
// (3 weights, 3 coordinates), and a piece inside every face is listed like
// one at its last face, since its share of the tet (bary_share, a
// double-float determinant) costs as much as a split and would run three
// times, for a few lanes each, in the split step.  The pool's last 8 places are
// for steps of one lane, so that none ever has to clip a piece by itself (in a
// pool of 66 that had happened 5386 times on a clustered 128^3 lattice, with
// a stack in local memory: 2.7 -> 2.2 ms of the kernel).
constexpr int kBaryPool = 66;    // pieces per warp pool
constexpr int kBaryLast = 66;    // pieces whose share is to be added, per warp
constexpr int kBaryPairs = 640;  // partial pairs a CTA lists

constexpr int kBaryRoom = kBaryPool - 8;  // what steps of several lanes may fill (see the split step)

static_assert(kBaryRoom >= 32 && kBaryLast >= 31 + 32, "a build step fits");

struct BaryPool {
    float v[24][kBaryPool];         // row 6 q + i: vertex q's weights (i = 0..2) and coordinates (3..5)
    uint32_t flags[kBaryPool];      // the vertices' inside flags, a byte each
    float last[16][kBaryLast];      // weights 3 q + i, then the vertices' coordinate along the last face's axis
    uint32_t last_meta[kBaryLast];  // inside mask (15: the whole piece) | upper face << 4 | owner << 8
    uint16_t owner[kBaryPool];      // the piece's pair
};

using BaryList = PairListOf<kBaryPairs>;

__device__ __forceinline__ void put_share(BaryPool &pool, int slot, const float p[24], int f, int mask, int owner)
{
    const unsigned ax = bit_mask(f < 2), ay = bit_mask(f < 4);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int i = 0; i < 3; ++i) pool.last[3 * q + i][slot] = p[6 * q + i];
        pool.last[12 + q][slot] = bit_sel(ax, p[6 * q + 3], bit_sel(ay, p[6 * q + 4], p[6 * q + 5]));
    }
    pool.last_meta[slot] = (uint32_t)(mask | ((f & 1) << 4) | (owner << 8));
}

__device__ __forceinline__ long long share_fixed(F2 c)
{
    return vol_fixed(c.hi) + vol_fixed(c.lo);
}

// As clip_pairs: build(j, x) writes the coordinates (3 per vertex) of pair
// j's tet; on return list.volume(j) of this warp's pairs are the cells'
// shares of the tet in fixed point 2^kVolShift.
template <typename Build>
__device__ __forceinline__ uint64_t clip_bary_pairs(BaryPool &pool, BaryList &list, int *next, int np, Build build)
{
    static_assert(kBaryPairs <= 64 * 32, "a bit per 32 pairs");
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1;
    int top = 0, nlast = 0;
    uint64_t taken = 0;
    bool more_pairs = np > 0;
    for (;;) {
        if (nlast >= 32 || (nlast && !top && !more_pairs)) {
            // the shares of up to 32 pieces, or of their inside parts
            const int n = min(nlast, 32), idx = nlast - 1 - lane;
            if (lane < n) {
                const uint32_t m = pool.last_meta[idx];
                float w[12];
#pragma unroll
                for (int i = 0; i < 12; ++i) w[i] = pool.last[i][idx];
                const F2 c = bary_share(w);
                const float frac = side_fraction(pool.last[12][idx], pool.last[13][idx], pool.last[14][idx],
                                                 pool.last[15][idx], m & 15, (m & 16) ? 1.f : 0.f);
                const F2 cut = f2_mul_f(c, frac);
                const bool whole = (m & 15) == 15;
                list.add((int)(m >> 8), share_fixed({whole ? c.hi : cut.hi, whole ? c.lo : cut.lo}));
            }
            nlast -= n;
            __syncwarp();
            continue;
        }
        if (top <= kBaryRoom - 32 && more_pairs) {
            // build step
            int j = 0;
            if (lane == 0) j = atomicAdd(next, 32);
            j = __shfl_sync(0xffffffffu, j, 0);
            more_pairs = j + 32 < np;
            if (j >= np) continue;
            taken |= 1ull << (j >> 5);
            const int nb = min(32, np - j);
            j += lane;
            float p[24];
            uint32_t flags = 0;
            int f = 0, mask = 0;
            bool push = false, share = false;
            if (lane < nb) {
                float x[12];
                build(j, x);
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        p[6 * q + i] = q == i + 1 ? 1.f : 0.f;  // the tet itself (bary_identity)
                        p[6 * q + 3 + i] = x[3 * q + i];
                    }
                flags = face_flags(x, x + 3, x + 6, x + 9);
                const int next = 63 & ~flags_all(flags);  // crossed, or entirely outside
                if ((63 & ~flags_any(flags)) == 0) {
                    push = (next & (next - 1)) != 0;
                    share = !push;
                    f = 31 - __clz(next | 1);
                    mask = next ? flags_mask(flags, f) : 15;
                }
                list.set(j, 0);
            }
            const unsigned pushing = __ballot_sync(0xffffffffu, push), lasts = __ballot_sync(0xffffffffu, share);
            if (push) {
                const int slot = top + __popc(pushing & lt);
#pragma unroll
                for (int x = 0; x < 24; ++x) pool.v[x][slot] = p[x];
                pool.flags[slot] = flags;
                pool.owner[slot] = (uint16_t)j;
            }
            if (share) put_share(pool, nlast + __popc(lasts & lt), p, f, mask, j);
            top += __popc(pushing);
            nlast += __popc(lasts);
            __syncwarp();
            continue;
        }
        if (!top) return taken;
        // split step: lane l takes slot top - 1 - l
        const int n = min(top, 32), idx = top - 1 - lane;
        int owner = 0;
        int code[3] = {0, 0, 0};  // per child: 0 dropped, 1 inside, 2 at its last face, 3 to split further
        uint32_t cflags[3];
        int cnext[3];
        float A[6], B[6], C[6], E[4][6];
        unsigned k1 = 0, k2 = 0;
        if (lane < n) {
            const uint32_t m = pool.flags[idx];
            owner = pool.owner[idx];
            const int left = 63 & flags_any(m);
            const int f = flags_face(m, left & ~flags_all(m)), mask = flags_mask(m, f);
            const int pm = split_perm(mask), k = split_kin(mask);
            const int ia = pm & 3, ib = (pm >> 2) & 3, ic = (pm >> 4) & 3, id = (pm >> 6) & 3;
            float D[6];
#pragma unroll
            for (int x = 0; x < 6; ++x) {
                A[x] = pool.v[6 * ia + x][idx];
                B[x] = pool.v[6 * ib + x][idx];
                C[x] = pool.v[6 * ic + x][idx];
                D[x] = pool.v[6 * id + x][idx];
            }
            const int ax = 3 + (f >> 1);
            cut_points<6>(A, B, C, D, pool.v[6 * ia + ax][idx], pool.v[6 * ib + ax][idx], pool.v[6 * ic + ax][idx],
                          pool.v[6 * id + ax][idx], k, f, E);
            k1 = bit_mask(k == 1);
            k2 = bit_mask(k == 2);
            const int keep = left & ~(1 << f);
            const unsigned keep4 = 0x01010101u * (unsigned)keep;
            const unsigned wV = __byte_perm(m & keep4, 0, ia + 16 * ib + 256 * ic);  // bytes A B C
            const unsigned wE = face_flags(E[0] + 3, E[1] + 3, E[2] + 3, E[3] + 3) & keep4;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                cflags[c] = __byte_perm(wV, wE, child_bytes(c, k1, k2));
                cnext[c] = keep & ~flags_all(cflags[c]);  // crossed, or entirely outside
                const bool out = (keep & ~flags_any(cflags[c])) != 0 || (c > 0 && k1);
                code[c] = out ? 0 : (cnext[c] == 0 ? 1 : ((cnext[c] & (cnext[c] - 1)) == 0 ? 2 : 3));
            }
        }
        unsigned sm[3], lm[3];  // the lanes whose child c goes to the pool / to the share list
        int ns = 0, nl = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sm[c] = __ballot_sync(0xffffffffu, code[c] == 3);
            lm[c] = __ballot_sync(0xffffffffu, code[c] == 1 || code[c] == 2);
            ns += __popc(sm[c]);
            nl += __popc(lm[c]);
        }
        // The first lanes whose children fit commit their step, as in
        // clip_pairs; several lanes fill kBaryRoom of the pool at most.  A
        // step by one lane always fits: a piece crossing 6 faces leaves at most
        // 2 pieces pending at each of the 4 splits before its last two, so
        // clipping it and then its children, last in first out, takes 8 more.
        int commit = n;
        if (top - n + ns > kBaryRoom || nlast + nl > kBaryLast) {
            int s_incl = 0, l_incl = 0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                s_incl += __popc(sm[c] & (lt << 1 | 1));
                l_incl += __popc(lm[c] & (lt << 1 | 1));
            }
            const unsigned bad = __ballot_sync(0xffffffffu, lane > 0 && lane < n && (top - (lane + 1) + s_incl > kBaryRoom ||
                                                                                     nlast + l_incl > kBaryLast));
            if (bad) commit = __ffs(bad) - 1;
            const unsigned cm = commit < 32 ? (1u << commit) - 1 : 0xffffffffu;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sm[c] &= cm;
                lm[c] &= cm;
            }
        }
        top -= commit;
        __syncwarp();  // every lane has read its slot
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (lane < commit && code[c]) {
                float ch[24];
                split_child<6>(c, k1, k2, A, B, C, E, ch);
                if (code[c] == 3) {
                    const int slot = top + __popc(sm[c] & lt);
#pragma unroll
                    for (int x = 0; x < 24; ++x) pool.v[x][slot] = ch[x];
                    pool.flags[slot] = cflags[c];
                    pool.owner[slot] = (uint16_t)owner;
                } else {
                    const int f = 31 - __clz(cnext[c] | 1);
                    put_share(pool, nlast + __popc(lm[c] & lt), ch, f, code[c] == 1 ? 15 : flags_mask(cflags[c], f), owner);
                }
            }
            top += __popc(sm[c]);
            nlast += __popc(lm[c]);
        }
        __syncwarp();
    }
}
#endif

}  // namespace adeco

// kernels.cuh -- the deposit kernels.
//
// Work decomposition: a deposit is a list of work items; an item pairs one
// output grid (a GridDesc: an octree leaf block, a zoom box, or the grid of a
// reference-boundary call) with one vertex block of at most 8^3 vertices
// (7^3 lattice cubes: a meta-cell of a resident lattice, or a sub-block of a
// reference-format patch).  A CTA stages the block's vertices in shared
// memory, culls its cubes against the grid box, and deposits the surviving
// tets 256 at a time, in phases that all its warps run together:
//   set-up     each warp builds the table entries of 32 tets, a lane each;
//   classify   the tets' candidate (tet, cell) pairs are flattened over the
//              CTA and classified with per-tet plane bounds; easy cells are
//              scattered at once, partial ones listed;
//   clip       the listed pairs are clipped by the warps' clip engines;
//   deposit    the listed pairs' masses are scattered, and the warps that are
//              through first take the pairs that one face cuts.
// Together, because the code of all the phases is larger than the SM's
// instruction cache: with each warp in a phase of its own (a warp taking 32
// tets through all of them) a third of the issue slots waited for
// instructions (no_instruction 2.9 stall cycles an issue; 0.25 in phases).
// And the pairs are the CTA's, so no warp waits for one that holds more.
//
// Mass is accumulated as 64-bit fixed point (2^shift units per mass unit)
// with integer atomics: the sum is exact and independent of the order in
// which tets land, so results are bit-reproducible run to run and the same
// whether a request runs alone or inside a batch.
#pragma once

#include "clip_engine.cuh"
#include "geometry.cuh"

namespace adeco {

// 8 warps per CTA and 2 CTAs per SM (16 warps, <= 128 registers, 2 x ~115 KB
// of shared memory): the staged vertex block (20 KB) is shared by 8 warps
// instead of 4, which leaves room for a fourth warp per scheduler.  Against 3
// CTAs of 4 warps (12 warps per SM) this is 5.6% faster on a 208^3 lattice;
// 8 warps per SM is 11% slower.
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxVerts = 512;   // 8^3
constexpr int kMaxCubes = 343;   // 7^3
constexpr int kWave = kThreads;       // tets set up together
constexpr int kQueue = 128;            // largest clip_batch: the whole pair list

struct Item {
    long long base;  // vertex index of the block origin (lattice) or of the patch origin + offset
    int grid;        // GridDesc index
    int nv;          // vertex counts vx | vy<<8 | vz<<16 (each <= 8)
};

enum SrcKind : int { SRC_LATTICE_F4 = 0, SRC_PATCH_F3 = 1 };

struct DepositParams {
    const Item *items;
    int n_items;
    int src_kind;
    const GridDesc *grids;
    const void *src;
    long long stride_y, stride_z;     // vertex strides of the source
    int order;                        // ORDER_REF or ORDER_CONFORMING
    int pad_check;                    // skip cubes with a 666 vertex (patch inputs)
    unsigned long long *out;          // fixed-point accumulators (mixed path)
    double *out_d;                    // FP64 grids (plain path)
    int *counter;                     // persistent work counter
    unsigned long long *stats;        // kNumStats counters or nullptr
    const int *nothing;               // null, or set when no tet can meet its grid: the launch ends at once
    int *error;                       // device error flag (bit 0: tet too large, bit 2: route list full,
                                      // bit 3: a bounded wait timed out; no deposit kernel has one)
    // ill-conditioned tets, deposited by a second launch (route_fp64_kernel):
    // entries item << 16 | (cube slot * 6 + tet), count in *route_count
    unsigned long long *route;
    unsigned long long *route_count;
    unsigned long long route_cap;
    // launch-shape and batching parameters (set by the host, tunable)
    int parts;           // CTAs that share an item, each with every parts-th cube (>= 1)
    int per_cta_items;   // items a CTA takes before it exits (0: persistent, until the queue is empty)
    int clip_batch;      // share of the pair list used, in kQueue-ths (64..kQueue)
};

enum Stat : int {
    ST_TETS = 0,         // tets with nonzero volume that meet the grid
    ST_CAND = 1,         // candidate pairs
    ST_BBOX = 2,         // pairs passing the AABB test
    ST_INSIDE = 3,       // TET_INSIDE_CELL pairs
    ST_CELLIN = 4,       // CELL_INSIDE_TET pairs
    ST_PARTIAL = 5,      // clipped pairs
    ST_FP64 = 6,         // pairs decided by the FP64 plane test
    ST_FALLBACK = 7,     // pieces clipped serially because the warp pool was full
    kNumStats = 8
};

// What the classification needs of N tets, in 16-byte words of shared memory:
// it reads 24 numbers of a pair's tet, and a load instruction each had been a
// tenth of its instructions.
template <int N>
struct TetPlanes {
    // inward face normals n and plane offsets d = n . (face centroid): inside
    // <=> n.x - d > 0.  Two faces at a time: (nx ny) of faces 0 and 1, (nz -d) of
    // them, then faces 2 and 3
    float4 plane[4][N];
    float4 lower[N];     // tet AABB in the anchor frame, minimum; FP32 error bound of the plane tests (largest face)
    float4 upper[N];     //   maximum; candidate extents of axes 0 | 1 << 16, as bits
    float f6[N];         // mass per unit of 6x clipped volume (tet mass / |6V| in cell units)
    uint16_t lo[3][N];   // anchor cell (first candidate cell) in grid indices (dims <= 4096)
};

// The vertices of up to 32 tets in their anchor cells' frames (cell units).
struct TetVertices {
    float q[12][32];    // rounded
    float qlo[12][32];  // rounding remainders: q + qlo carries the vertex to ~44 bits
};

// A table with everything in it, the exact plane offsets' remainders too
// (d + dlo: ~44 bits), which setup_tet<true> stores.  The kernels form the
// vertices and the exact offsets again for the pairs that need them.
struct WarpTets : TetPlanes<32>, TetVertices {
    static constexpr bool kHasRest = true;
    float dlo[4][32];
    uint16_t ex[3][32];  // candidate extents (cells per axis)
};

ADECO_HD inline void tet_coord(const WarpTets &W, const GridDesc &, int s, int v, int x, float &hi, float &lo)
{
    hi = W.q[3 * v + x][s];
    lo = W.qlo[3 * v + x][s];
}

// Tets whose conditioning kappa = (longest edge)^3 / |6V| exceeds this take
// the FP64 route: FP32 vertices in the cell frame carry ~2^-24 * kappa
// relative error into every cell fraction, so a flat tet (kappa >> 1) would
// miss the 1e-5 per-cell bar.  Lattice tets sit near kappa = 5.2.
constexpr float kKappaFp64 = 32.f;

// Waits, sleeping `ns` between looks, until *count is 0, at most `limit`
// looks; false if the limit ran out first.  A spin-wait in a kernel goes
// through here, so that none can wait forever (the deposit kernels have none).
__device__ __forceinline__ bool wait_zero_bounded(const int *count, unsigned limit, unsigned ns)
{
    for (unsigned spin = 0; *(volatile const int *)count != 0; ++spin) {
        if (spin >= limit) return false;
        __nanosleep(ns);
    }
    return true;
}

// A tet of the wave has more than 1024 candidate cells along an axis; a warp
// has more than kMaxPartPairs / kWarps candidate pairs.
constexpr int kWideTet = 1, kManyPairs = 2;

// The staged vertex block and the wave's tets.
struct WaveTets : TetPlanes<kWave> {
    static constexpr bool kHasRest = false;
    float gh[3][kMaxVerts];  // grid-frame coordinates of the staged vertices, hi
    float gl[3][kMaxVerts];  //   and lo parts
    ushort4 vid[kWave];      // the tets' vertices, ordered by the orientation rule
};

// Vertex coordinate of a wave's tet in its anchor cell's frame: formed again
// from the staged vertex with the operations of the set-up.
__device__ __forceinline__ void tet_coord(const WaveTets &W, const GridDesc &g, int s, int v, int x, float &hi, float &lo)
{
    const ushort4 id = W.vid[s];
    const int i = v == 0 ? id.x : (v == 1 ? id.y : (v == 2 ? id.z : id.w));
    shift_frame(W.gh[x][i], W.gl[x][i], W.lo[x][s], g.drcell[x], hi, lo);
}

// the same of vertices v and w
__device__ __forceinline__ void tet_coord2(const WaveTets &W, const GridDesc &g, int s, int v, int w, int x, float2 &hi,
                                           float2 &lo)
{
    const ushort4 id = W.vid[s];
    const int i = v == 0 ? id.x : (v == 1 ? id.y : (v == 2 ? id.z : id.w));
    const int j = w == 0 ? id.x : (w == 1 ? id.y : (w == 2 ? id.z : id.w));
    shift_frame2(make_float2(W.gh[x][i], W.gh[x][j]), make_float2(W.gl[x][i], W.gl[x][j]), (float)W.lo[x][s], g.drcell[x],
                 hi, lo);
}

struct SharedMixed {
    WaveTets wt;
    uint2 range[kMaxVerts];   // the staged vertices' candidate cells and box flags (vertex_range)
    alignas(16) int src_off[6][4];        // the six tets' corners: offsets in the source from a cube's first vertex
    alignas(8) uint16_t vert_off[6][4];  //   and among the staged vertices
    uint16_t cubes[kMaxCubes + 1];  // the live cubes' first staged vertices
    int n_cubes;
    int item, part;
    GridDesc g;
    // per warp, its tets that have pairs, in order: the tet, and the warp's
    // pairs before it (INT_MAX past the last)
    int start[kWave];
    uint8_t tet[kWave];
    int warp_pairs[kWarps];
    int all_pairs[kWarps], part_end;  // of a wave taken in parts: its warps' pairs, the warps taken (wave_next_part)
    int cursor;          // first candidate pair of the wave not yet taken
    int cut[2];          // one-face pairs at the list's end (alternating as list.n),
    int cut_next[2];     //   and the first not taken
    int flags[2];        // of the wave (even, odd): kWideTet, kManyPairs
    PairList list;
    WarpPool pool[kWarps];
};

__device__ __forceinline__ void stat_add(unsigned long long *stats, int which, unsigned long long v)
{
    if (stats && v) atomicAdd(stats + which, v);
}

// warp-wide sum of a per-lane count, added once per warp
__device__ __forceinline__ void warp_stat(unsigned long long *stats, int which, unsigned v)
{
    if (!stats) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) stat_add(stats, which, v);
}

// ---------------------------------------------------------------- staging
// What the candidate range of a tet needs of each vertex, once per vertex
// instead of once per tet (2058 tets share 512 vertices, and the six FP32
// divisions of candidate_range were a fifth of the set-up): per axis twice
// the floor of (x - gmin) / delta, x limited to the grid box, plus one where
// it is no whole number.  The word grows with x, so a tet's first and last
// candidate cells (candidate_range) come from the least and the greatest word
// of its vertices.  x: axes 0 | 1 << 16; y: axis 2 | flags << 16.
constexpr uint32_t kBelowMax = 0x7u << 16, kAboveMin = 0x38u << 16;    // x < gmax, gmin < x, a bit per axis
constexpr uint32_t kCullBox = 0xfc0u << 16, kPadVertex = 0x1000u << 16;  // the same two for the cull box; padding

ADECO_HD inline uint2 vertex_range(const float p[3], const GridDesc &g, bool pad)
{
    uint32_t w[3], flags = pad ? kPadVertex : 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float x = p[a];
        const float lim = (x < g.gmin[a]) ? g.gmin[a] : x;
        const float q = div_rn(sub_rn((lim < g.gmax[a]) ? lim : g.gmax[a], g.gmin[a]), g.delta[a]);
        int lo = (int)floorf(q);
        const int more = (int)ceilf(q) > lo;
        lo = lo < 0 ? 0 : (lo > 8191 ? 8191 : lo);
        w[a] = (uint32_t)(2 * lo + more);
        flags |= ((x < g.gmax[a] ? 1u : 0u) | (g.gmin[a] < x ? 8u : 0u) | (x < g.cull_max[a] ? 64u : 0u) |
                  (g.cull_min[a] < x ? 512u : 0u)) << (16 + a);
    }
    return make_uint2(w[0] | (w[1] << 16), w[2] | flags);
}

// A tet's candidate cells [lo, hi] along axis a, in grid indices up to top, from
// the least and the greatest words of its vertices.
ADECO_HD inline void word_range(uint2 mn, uint2 mx, int a, int top, int &lo, int &hi)
{
    const int wlo = (int)((a == 2 ? mn.y : (mn.x >> (16 * a))) & 0xffffu),
              whi = (int)((a == 2 ? mx.y : (mx.x >> (16 * a))) & 0xffffu);
    lo = wlo >> 1;
    hi = (whi + 1) >> 1;
    lo = lo > top ? top : lo;
    hi = hi > top ? top : hi;
}

// position of source vertex gi (the w of a lattice vertex is not used)
__device__ __forceinline__ float3 load_vertex(const DepositParams &P, long long gi)
{
    if (P.src_kind == SRC_LATTICE_F4) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(P.src) + gi);
        return make_float3(q.x, q.y, q.z);
    }
    const float *s = reinterpret_cast<const float *>(P.src) + 3 * gi;
    return make_float3(__ldg(s), __ldg(s + 1), __ldg(s + 2));
}

// vertex v < 512 of a block vx vertices wide (<= 8) -> v / vx, exact
__device__ __forceinline__ int small_div(int v, int vx) { return (int)((unsigned)(v * (65536 / vx + 1)) >> 16); }

__device__ __forceinline__ void stage_block(const DepositParams &P, const Item &it, const GridDesc &g, SharedMixed &S,
                                            int vx, int vy, int vz)
{
    const int nvt = vx * vy * vz;
    for (int v = threadIdx.x; v < nvt; v += blockDim.x) {
        const int r = small_div(v, vx), i = v - r * vx, k = small_div(r, vy), j = r - k * vy;
        const float3 q = load_vertex(P, it.base + i + P.stride_y * j + P.stride_z * k);
        const float p[3] = {q.x, q.y, q.z};
        bool pad = false;
        if (P.pad_check) {
            // the reference's padding test on the float inputs
            const float sum = __fadd_rn(__fadd_rn(fabsf(__fsub_rn(p[0], 666.f)), fabsf(__fsub_rn(p[1], 666.f))),
                                        fabsf(__fsub_rn(p[2], 666.f)));
            pad = (double)sum < 1.E-03;
        }
        S.range[v] = vertex_range(p, g, pad);
#pragma unroll
        for (int a = 0; a < 3; ++a) grid_frame(p[a], g.gmin[a], g.scale_hi[a], g.scale_lo[a], S.wt.gh[a][v], S.wt.gl[a][v]);
    }
    if (threadIdx.x < 24) {
        const int t = threadIdx.x >> 2, q = threadIdx.x & 3;
        const int3 o = corner_offset(P.order, tet_conn(t, q));
        S.vert_off[t][q] = (uint16_t)(o.x + vx * (o.y + vy * o.z));
        S.src_off[t][q] = (int)(o.x + P.stride_y * o.y + P.stride_z * o.z);
    }
}

// cube whose first staged vertex is v0: alive if no padding vertex and its
// AABB strictly overlaps the grid box (the tile's widened box)
__device__ __forceinline__ bool cube_alive(const SharedMixed &S, int v0, int vx, int vy)
{
    uint32_t f = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) f |= S.range[v0 + (s & 1) + vx * (((s >> 1) & 1) + vy * (s >> 2))].y;
    return (f & (kCullBox | kPadVertex)) == kCullBox;
}

// ------------------------------------------------------ per-tet set-up
// Candidate pairs of one tet are limited to kMaxPairsPerTet, so that a pair's
// number within its tet leaves the top bits of a list entry free and a warp's
// 32 tets have at most 2^30 of them; a larger tet sets the error flag and is
// skipped.
constexpr long long kMaxPairsPerTet = 1LL << 25;

// The pairs of a wave's tets are numbered through in an int, but those of its
// 8 warps may be 2^33 (tets that each cover a grid of hundreds of cells an
// axis).  They are taken in parts: the warps [first, end) whose pairs together
// stay below 2^31, the 32 that each warp may add to the cursor past the end
// among them.  Returns end > first; total: the part's pairs.  A wave without
// kManyPairs is one part and does not ask (asking took 0.6% of the time of
// octree leaves).
constexpr int kMaxPartPairs = INT_MAX - 32 * kWarps;
static_assert(32 * kMaxPairsPerTet <= kMaxPartPairs, "a warp's pairs fit a part");

ADECO_HD inline int wave_part(const int *warp_pairs, int first, int &total)
{
    int end = first;
    total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const bool take = w == end && warp_pairs[w] <= kMaxPartPairs - total;
        total += take ? warp_pairs[w] : 0;
        end += take;
    }
    return end;
}

// Offset of a tet face's plane n . x = d through the face's centroid, from
// its vertices as FP32 pairs (hi + lo) and the FP32 normal n: 3 d = n . (va
// + vb + vc) in double-float, divided by 3 as a product with 1/3 whose
// remainder (exact, fma) is carried into the low part, so that d_hi + d_lo
// keeps ~44 bits.  kStored: both products rounded, as if the offset had been
// stored (else the compiler may contract them into the sums they go to).
template <bool kStored = false>
ADECO_HD inline F2 plane_offset(const float qa[3], const float la[3], const float qb[3], const float lb[3],
                                const float qc[3], const float lc[3], const float n[3])
{
    F2 dd = {0.f, 0.f};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const F2 sum = f2_add(f2_add(F2{qa[a], la[a]}, F2{qb[a], lb[a]}), F2{qc[a], lc[a]});
        dd = f2_add(dd, f2_mul_f(sum, n[a]));
    }
    constexpr float kThird = 1.f / 3.f;
    if constexpr (kStored) {
        const float d_hi = mul_rn(dd.hi, kThird);
        return {d_hi, mul_rn(fmaf(-d_hi, 3.f, dd.hi) + dd.lo, kThird)};
    }
    const float d_hi = dd.hi * kThird;
    return {d_hi, (fmaf(-d_hi, 3.f, dd.hi) + dd.lo) * kThird};
}

// Entry t of table W from the grid-frame coordinates of a tet's vertices,
// ordered by the orientation rule (frame(q, a, hi, lo): vertex q, axis a), and
// its candidate cells as vertex_range words (mn / mx: the least and the
// greatest of its vertices).  Returns the candidate pair count (0 if the tet
// is skipped); *wide: more than 1024 of them along an axis.
//
// kExactD: each face's plane offset in double-float, rounded once (d; its
// remainder too where the table has room for it, dlo).  Otherwise an FP32 d,
// whose rounding the classification's error band covers.  The double-float
// offsets had been ~40% of the set-up: octree leaves and boundary grids do
// without, zoom grids, whose tets have thousands of pairs each, use them.
// The one-face closed form takes exact offsets either way (it forms them from
// the stored vertices).
template <bool kExactD, class Table, class Frame>
ADECO_HD inline int setup_frame(uint2 mn, uint2 mx, Frame frame, const GridDesc &g, Table &W, int t, int *error,
                                bool *fp64_route, bool *wide)
{
    long long cnt0 = 1;
    unsigned cnt = 1;
    float R = 0.f, bmin[3], bmax[3];
    float V[4][3], L[4][3];  // the vertices in the anchor frame, hi and lo
    uint32_t ext01 = 0;
    int big_ex = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int lo, hi;
        word_range(mn, mx, a, g.dims - 1, lo, hi);
        lo = lo < g.tile_lo[a] ? g.tile_lo[a] : lo;
        hi = hi > g.tile_hi[a] ? g.tile_hi[a] : hi;
        cnt0 = hi < lo ? 0 : cnt0 * (hi - lo + 1);
        // Tight range: of the candidate cells [lo, hi], only those whose box
        // [c r, c r + 1] (grid frame) meets the tet's AABB can receive mass (the
        // rest fail the AABB test).  Bounds widened by the FP32 rounding of the
        // grid-frame coordinates; the frame is then anchored at the first cell.
        float h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) frame(q, a, h[q], l[q]);
        const float bmn = fminf(fminf(h[0], h[1]), fminf(h[2], h[3])), bmx = fmaxf(fmaxf(h[0], h[1]), fmaxf(h[2], h[3]));
        const float ir = g.inv_rcell_f[a];
        const float m0 = 4e-7f * (fabsf(bmn) + 2.f), m1 = 4e-7f * (fabsf(bmx) + 2.f);
        const int u0 = (int)floorf((bmn - 1.f) * ir - m0) + 1, u1 = (int)ceilf(bmx * ir + m1) - 1;
        const int c0 = lo > u0 ? lo : u0, c1 = hi < u1 ? hi : u1;
        const int ex = c1 - c0 + 1;
        cnt = ex > 0 ? cnt * (unsigned)ex : 0u;
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            float2 hi, lo2;
            shift_frame2(make_float2(h[q], h[q + 1]), make_float2(l[q], l[q + 1]), (float)c0, g.drcell[a], hi, lo2);
            V[q][a] = hi.x;
            V[q + 1][a] = hi.y;
            L[q][a] = lo2.x;
            L[q + 1][a] = lo2.y;
        }
        R = fmaxf(R, (float)(ex - 1) + 1.f);
        bmin[a] = fminf(fminf(V[0][a], V[1][a]), fminf(V[2][a], V[3][a]));
        bmax[a] = fmaxf(fmaxf(V[0][a], V[1][a]), fmaxf(V[2][a], V[3][a]));
        R = fmaxf(R, fmaxf(fabsf(bmin[a]), fabsf(bmax[a])));
        if constexpr (Table::kHasRest) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                W.q[3 * q + a][t] = V[q][a];
                W.qlo[3 * q + a][t] = L[q][a];
            }
        }
        if (a < 2) ext01 |= (uint32_t)(ex & 0xffff) << (16 * a);
        W.lo[a][t] = (uint16_t)c0;
        big_ex = big_ex > ex ? big_ex : ex;
        if constexpr (Table::kHasRest) W.ex[a][t] = (uint16_t)ex;
    }
    if (cnt0 > kMaxPairsPerTet) {
#ifdef __CUDA_ARCH__
        if (error) atomicOr(error, 1);
#else
        if (error) *error |= 1;
#endif
        return 0;
    }
    if (cnt0 <= 0 || cnt == 0) return 0;
    // |6 V| in the anchor frame from the FP32 pairs, in double-float (the
    // tet's volume normaliser): edge vectors from vertex 3, then the triple
    // product with TwoProd / TwoSum, a cofactor of the first edge at a time
    F2 w6 = {0.f, 0.f};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = a == 2 ? 0 : a + 1, c = a == 0 ? 2 : a - 1;
        auto edge = [&](int q, int x) {
            return f2_add(F2{V[q][x], L[q][x]}, F2{-V[3][x], -L[3][x]});
        };
        const F2 cof = f2_add(f2_mul(edge(1, b), edge(2, c)), f2_neg(f2_mul(edge(1, c), edge(2, b))));
        w6 = f2_add(w6, f2_mul(edge(0, a), cof));
    }
    if (w6.hi < 0.f) w6 = f2_neg(w6);
    const float vq6 = w6.hi;
    W.f6[t] = f2_div_to_f(F2{g.mf_hi, g.mf_lo}, w6);  // mass per unit of 6x volume
    // planes from the FP32 vertices: inward normals (outward ones negated:
    // faces (0,1,2) (0,2,3) (0,3,1) (1,3,2)); each plane's offset is taken
    // through the face's centroid, so that the FP32 rounding of the normal
    // only turns the plane about the centroid (the one-face closed form
    // relies on it)
    // edges v1 - v0, v2 - v0, v3 - v0, v2 - v1, v3 - v1 and the largest of their components
    constexpr int kFrom[6] = {0, 0, 0, 1, 1, 2}, kTo[6] = {1, 2, 3, 2, 3, 3};
    float e[5][3], big[5], normal[4][4], tolmax = 0.f, L2 = 0.f;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        float d[3], sq = 0.f;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            d[x] = V[kTo[k]][x] - V[kFrom[k]][x];
            sq = fmaf(d[x], d[x], sq);
            if (k < 5) e[k][x] = d[x];
        }
        if (k < 5) big[k] = fmaxf(fmaxf(fabsf(d[0]), fabsf(d[1])), fabsf(d[2]));
        L2 = fmaxf(L2, sq);
    }
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        // n_in = (vb - va) x (vc - va) with the outward order reversed: faces (0,2,1) (0,3,2) (0,1,3) (1,2,3)
        constexpr int kA[4] = {0, 0, 0, 1}, kB[4] = {2, 3, 1, 2}, kC[4] = {1, 2, 3, 3};
        constexpr int kE1[4] = {1, 2, 0, 3}, kE2[4] = {0, 1, 2, 4};
        const float *A = V[kA[f]], *B = V[kB[f]], *C = V[kC[f]], *e1 = e[kE1[f]], *e2 = e[kE2[f]];
        const float nn[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
        float offset;
        if constexpr (kExactD) {
            const F2 d = plane_offset(A, L[kA[f]], B, L[kB[f]], C, L[kC[f]], nn);
            offset = d.hi;
            if constexpr (Table::kHasRest) W.dlo[f][t] = d.lo;
        } else {
            constexpr float kThird = 1.f / 3.f;
            offset = (nn[0] * (A[0] + B[0] + C[0]) + nn[1] * (A[1] + B[1] + C[1]) + nn[2] * (A[2] + B[2] + C[2])) * kThird;
        }
        normal[f][0] = nn[0];
        normal[f][1] = nn[1];
        normal[f][2] = nn[2];
        normal[f][3] = -offset;
        // generous bound on the FP32 rounding of n.x - d (|x| <= R + 1)
        tolmax = fmaxf(tolmax, 1.0e-5f * big[kE1[f]] * big[kE2[f]] * (R + 1.f));
    }
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const int k = f & 2, i = 2 * (f & 1);
        W.plane[f][t] = make_float4(normal[k][i], normal[k + 1][i], normal[k][i + 1], normal[k + 1][i + 1]);
    }
    W.lower[t] = make_float4(bmin[0], bmin[1], bmin[2], tolmax);
    W.upper[t] = make_float4(bmax[0], bmax[1], bmax[2], u2f(ext01));
    // conditioning: longest edge cubed over |6V|, both in cell units.  L^3 <=
    // kappa |6V| squared (both sides non-negative): no square root; NaN or an
    // overflow routes the tet
    *wide = big_ex > 1024;
    *fp64_route = !(L2 * L2 * L2 <= (kKappaFp64 * kKappaFp64) * (vq6 * vq6));
    return (int)cnt;
}

// One tet from its positions (bit-exact orientation rule and candidate range)
// and their grid-frame coordinates.
template <bool kExactD = true, class Table>
ADECO_HD inline int setup_tet(const float3 v[4], const float gh[4][3], const float gl[4][3], const GridDesc &g,
                              Table &W, int lane, int *error, bool *fp64_route)
{
    *fp64_route = false;
    bool wide;
    const int sgn = vol6_sign_ref(vol6_exact(v[0], v[1], v[2], v[3]));
    int lo[3], hi[3];
    if (!candidate_range(v, g, lo, hi) || sgn == 0) return 0;
    const uint2 mn = make_uint2((uint32_t)(2 * lo[0] | (2 * lo[1]) << 16), (uint32_t)(2 * lo[2]));
    const uint2 mx = make_uint2((uint32_t)(2 * hi[0] | (2 * hi[1]) << 16), (uint32_t)(2 * hi[2]));
    return setup_frame<kExactD>(
        mn, mx,
        [&](int q, int a, float &h, float &l) {
            const int v_ = (sgn < 0 && (q == 0 || q == 3)) ? 3 - q : q;  // swap 0 <-> 3 when negative
            h = gh[v_][a];
            l = gl[v_][a];
        },
        g, W, lane, error, fp64_route, &wide);
}

// face f's normal and -d
template <class Table>
ADECO_HD inline float4 face_plane(const Table &W, int f, int s)
{
    const float *p = &W.plane[f & 2][s].x + (f & 1), *q = &W.plane[(f & 2) + 1][s].x + (f & 1);
    return make_float4(p[0], p[2], q[0], q[2]);
}

enum PairClass : int { P_NO = 0, P_TET_INSIDE = 1, P_CELL_INSIDE = 2, P_PARTIAL = 3 };

// FP64 evaluation of the four plane bounds for a cell whose FP32 test was
// inside the error band: exact decision for the FP32-rounded tet.
template <class Table>
ADECO_HD
#ifdef __CUDA_ARCH__
__noinline__
#endif
int classify_fp64(const Table &W, const GridDesc &g, int s, int a, int b, int c)
{
    const double ca = a * g.rcell[0], cb = b * g.rcell[1], cc = c * g.rcell[2];
    double q[4][3];
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            float hi, lo;
            tet_coord(W, g, s, v, x, hi, lo);
            q[v][x] = (double)hi + (double)lo;
        }
    const int fa[4] = {0, 0, 0, 1}, fb[4] = {2, 3, 1, 2}, fc[4] = {1, 2, 3, 3};
    bool all_in = true;
    for (int f = 0; f < 4; ++f) {
        const double e1x = q[fb[f]][0] - q[fa[f]][0], e1y = q[fb[f]][1] - q[fa[f]][1], e1z = q[fb[f]][2] - q[fa[f]][2];
        const double e2x = q[fc[f]][0] - q[fa[f]][0], e2y = q[fc[f]][1] - q[fa[f]][1], e2z = q[fc[f]][2] - q[fa[f]][2];
        const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
        const double base = nx * (ca - q[fa[f]][0]) + ny * (cb - q[fa[f]][1]) + nz * (cc - q[fa[f]][2]);
        const double mx = base + fmax(nx, 0.0) + fmax(ny, 0.0) + fmax(nz, 0.0);
        const double mn = base + fmin(nx, 0.0) + fmin(ny, 0.0) + fmin(nz, 0.0);
        if (mx <= 0.0) return P_NO;
        all_in = all_in && (mn > 0.0);
    }
    return all_in ? P_CELL_INSIDE : P_PARTIAL;
}

// cross: the one tet face plane the cell straddles when the cell is certainly
// inside the other three (then cell ∩ tet = cell ∩ that face's half-space),
// else -1.
template <class Table>
ADECO_HD inline int classify_pair(const Table &W, const GridDesc &g, int s, int a, int b, int c, bool &used_fp64,
                                  int &cross)
{
    cross = -1;
    const float fa = (float)a, fb = (float)b, fc = (float)c;
    const float4 mn = W.lower[s], mx = W.upper[s];
    // strict AABB overlap with the cell [a,a+1] x [b,b+1] x [c,c+1]
    if (!(mn.x < fa + 1.f && fa < mx.x && mn.y < fb + 1.f && fb < mx.y && mn.z < fc + 1.f && fc < mx.z)) return P_NO;
    if (mn.x >= fa && mx.x <= fa + 1.f && mn.y >= fb && mx.y <= fb + 1.f && mn.z >= fc && mx.z <= fc + 1.f)
        return P_TET_INSIDE;
    bool all_in = true, unsure = false;
    int ncross = 0, fcross = 0;
    const float t = mn.w;
#pragma unroll
    for (int f = 0; f < 4; f += 2) {
        const float4 p = W.plane[f][s], q = W.plane[f + 1][s];
        const float2 nx = make_float2(p.x, p.y), ny = make_float2(p.z, p.w), nz = make_float2(q.x, q.y);
        const float2 base = fma2(nx, both(fa), fma2(ny, both(fb), fma2(nz, both(fc), make_float2(q.z, q.w))));
        const float2 pos = add2(add2(make_float2(fmaxf(nx.x, 0.f), fmaxf(nx.y, 0.f)),
                                     make_float2(fmaxf(ny.x, 0.f), fmaxf(ny.y, 0.f))),
                                make_float2(fmaxf(nz.x, 0.f), fmaxf(nz.y, 0.f)));
        const float2 mx2 = add2(base, pos), mn2 = add2(base, sub2(add2(add2(nx, ny), nz), pos));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float mx = i ? mx2.y : mx2.x, mn = i ? mn2.y : mn2.x;
            if (mx < -t) return P_NO;
            if (mx <= t) unsure = true;
            if (mn > t) continue;
            all_in = false;
            ++ncross;
            fcross = f + i;
            if (mn > -t) unsure = true;
        }
    }
    if (unsure) {
        used_fp64 = true;
        return classify_fp64(W, g, s, a, b, c);
    }
    if (ncross == 1) cross = fcross;
    return all_in ? P_CELL_INSIDE : P_PARTIAL;
}

// Value at the origin of cell (a, b, c) of face f's linear function G(u) =
// n . (cell origin + u - centroid), taken about the face's centroid so that
// the FP32 rounding of its normal only turns the plane about the centroid:
// the volume a slightly turned plane adds on one side of the centroid it
// removes on the other, and the tet's mass stays conserved over its cells.
// n . origin - (d + dlo) cancels terms as large as the tet is wide in cells:
// it is formed exactly in double-float (TwoProd of n with the integer cell
// offsets) and kept as a pair for the corner values.
template <bool kExactD = true, bool kStored = false, class Table>
ADECO_HD inline F2 face_value_at_cell(const Table &W, const GridDesc &g, int s, int a, int b, int c, int f)
{
    const int cc[3] = {a, b, c};
    const float4 pl = face_plane(W, f, s);
    const float n[3] = {pl.x, pl.y, pl.z};
    F2 G;
    if constexpr (kExactD) {
        G = {pl.w, -W.dlo[f][s]};
    } else {  // the exact offset setup_tet<true> would have stored
        const int fa = f == 3 ? 1 : 0, fb = f == 0 ? 2 : (f == 1 ? 3 : (f == 2 ? 1 : 2)),
                  fc = f == 0 ? 1 : (f == 1 ? 2 : 3);
        float q[3][3], l[3][3];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
#ifdef __CUDA_ARCH__
            if constexpr (!Table::kHasRest) {  // two vertices at a time
                float2 hi, lo;
                tet_coord2(W, g, s, fa, fb, x, hi, lo);
                q[0][x] = hi.x;
                q[1][x] = hi.y;
                l[0][x] = lo.x;
                l[1][x] = lo.y;
                tet_coord(W, g, s, fc, x, q[2][x], l[2][x]);
                continue;
            }
#endif
            tet_coord(W, g, s, fa, x, q[0][x], l[0][x]);
            tet_coord(W, g, s, fb, x, q[1][x], l[1][x]);
            tet_coord(W, g, s, fc, x, q[2][x], l[2][x]);
        }
        const F2 d = plane_offset<kStored>(q[0], l[0], q[1], l[1], q[2], l[2], n);
        G = {-d.hi, -d.lo};
    }
    float small = 0.f;  // the cells' deviation from unit size: n_x c_x dr_x, tiny
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const float fc = (float)cc[x];
        G = f2_add(G, f2_two_prod(n[x], fc));
        small = fmaf(n[x] * fc, g.drcell[x], small);
    }
    return f2_norm(G.hi, G.lo + small);
}

// 6x volume of cell (a, b, c) ∩ slot s's tet when the cell straddles only
// face f: the cube's part on its inside.
template <bool kExactD = true, bool kStored = false, class Table>
#ifdef __CUDA_ARCH__
__device__ __noinline__
#else
inline
#endif
float halfspace_pair_vol6(const Table &W, const GridDesc &g, int s, int a, int b, int c, int f)
{
    const float4 n = face_plane(W, f, s);
    return halfspace_cube_vol6(face_value_at_cell<kExactD, kStored>(W, g, s, a, b, c, f), n.x, n.y, n.z);
}

// Non-negative mass of a pair (FP32, about 1e-7 relative) -> the cell's
// 64-bit fixed-point accumulator, with integer operations only.  Inlined: as
// a call it made the pair loop save and restore its live registers in local
// memory around every scatter (C2: 16% of the kernel time).
__device__ __forceinline__ void scatter(const DepositParams &P, const GridDesc &g, const WaveTets &W, int s, int a,
                                        int b, int c, float m)
{
    const unsigned long long fx = to_fixed(m, g.shift);
    if (fx == 0ull) return;
    const long long i = W.lo[0][s] + a, j = W.lo[1][s] + b, k = W.lo[2][s] + c;
    const long long idx = g.out_offset + i + (long long)g.dims * (j + (long long)g.dims * k);
    atomicAdd(P.out + idx, fx);
}

#ifdef __CUDACC__
// scatter of whole tets' mass by lanes `lanes` of the warp: of those that add
// to the same cell, one adds for all (the same sum, in integers).  On grids
// coarser than the tets nearly every pair is a whole tet, and the additions to
// a few cells wait for one another: a 256^3 lattice onto 16^3 / 8^3 / 4^3 cells
// 12.9 / 25.3 / 33.3 ms lane by lane, 6.5 / 6.3 / 5.5 so.  Fewer than 12 lanes
// seldom share a cell and add by themselves.
__device__ __forceinline__ void scatter_whole(const DepositParams &P, const GridDesc &g, const WaveTets &W, int s, int a,
                                              int b, int c, unsigned lanes)
{
    unsigned long long fx = to_fixed(g.tet_mass, g.shift);
    const long long i = W.lo[0][s] + a, j = W.lo[1][s] + b, k = W.lo[2][s] + c;
    const long long idx = g.out_offset + i + (long long)g.dims * (j + (long long)g.dims * k);
    if (__popc(lanes) >= 12) {
        const unsigned same = __match_any_sync(lanes, idx);
        if ((int)(threadIdx.x & 31) != __ffs(same) - 1) return;
        fx *= (unsigned)__popc(same);
    }
    if (fx) atomicAdd(P.out + idx, fx);
}
#endif

// A pair's 6x volume, summed in fixed point 2^kVolShift (0 <= vacc < 2^59),
// times the tet's mass per unit of 6x volume.  The sum is converted to FP32
// with one rounding from two exact 24-bit parts (bits 35..58 and 11..34): the
// fma rounds their exact sum to nearest.  Rounding the upper part alone would
// drop the lower bits first -- a truncation, a bias of -6e-9 relative that
// showed in the total mass.  Bits 0..10 (below 3e-14 of a tet's 6x volume)
// are left out.
ADECO_HD inline float pair_mass(long long vacc, float f6)
{
    const float hi = (float)(int)(vacc >> 35), mid = (float)(int)((vacc >> 11) & 0xffffff);
    const float v = fmaf(hi, 0x1p35f, mid * 0x1p11f);
    return v * (f6 * 0x1p-56f);
}

// Tet of slot s in the frame of its candidate cell (a, b, c), as the clip
// engine takes it.  Along an axis whose lower face the tet does not reach,
// the cell's mirrored frame is used, so that the face it crosses lies at 0:
// a thin slice under the upper face otherwise lost ~6e-8 cell units per
// vertex (up to 5e-5 of such a cell's mass on a 256^3 lattice; 5e-7
// mirrored).  An odd number of reflections is undone by swapping vertices 0
// and 1 (the engine wants a positively oriented tet).
template <class Table>
ADECO_HD inline void piece_coords(const Table &W, const GridDesc &g, int s, int a, int b, int c, float p[12])
{
    const int cc[3] = {a, b, c};
    const float4 mn = W.lower[s];
    const float lower[3] = {mn.x, mn.y, mn.z};
    int nflip = 0;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const bool flip = lower[x] > (float)cc[x];
        nflip += flip;
#ifdef __CUDA_ARCH__
        if constexpr (!Table::kHasRest) {  // two vertices at a time
            float2 hi, lo;
#pragma unroll
            for (int v = 0; v < 4; v += 2) {
                tet_coord2(W, g, s, v, v + 1, x, hi, lo);
                const float2 c2 = cell_coord_fast2(hi, lo, cc[x], g.drcell[x], flip);
                p[3 * v + x] = c2.x;
                p[3 * v + 3 + x] = c2.y;
            }
            continue;
        }
#endif
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            float hi, lo;
            tet_coord(W, g, s, v, x, hi, lo);
            p[3 * v + x] = cell_coord_fast(hi, lo, cc[x], g.drcell[x], flip);
        }
    }
    const unsigned odd = bit_mask(nflip & 1);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const float t = p[x];
        p[x] = bit_sel(odd, p[3 + x], t);
        p[3 + x] = bit_sel(odd, t, p[3 + x]);
    }
}

#ifdef __CUDACC__
// Cell n of a box ex0 x ex1 cells wide, x fastest
__device__ __forceinline__ int3 box_cell(int ex0, int ex1, int n)
{
    int r, c;
    if (n < (1 << 20)) {
        // The quotient of n + 1/2 is at least 1 / (2 ex) away from a whole
        // number, the product with the approximate reciprocal closer than
        // n / ex 2^-22 to it: rounding down is exact.
        r = (int)(((float)n + 0.5f) * rcp_approx((float)ex0));
        c = (int)(((float)r + 0.5f) * rcp_approx((float)ex1));
    } else {
        r = n / ex0;
        c = r / ex1;
    }
    return make_int3(n - r * ex0, r - c * ex1, c);
}

// The cell of a candidate pair as PairList holds it: its offsets in the tet's
// candidate box, a | b << 10 | c << 20; in a wave with a box of more than 1024
// cells along an axis, the flattened offset.
__device__ __forceinline__ int3 flat_cell(const WaveTets &W, int s, int local)
{
    const uint32_t e = __float_as_uint(W.upper[s].w);
    return box_cell((int)(e & 0xffffu), (int)(e >> 16), local);
}
__device__ __forceinline__ int3 pair_cell(const WaveTets &W, int s, uint32_t e, bool wide)
{
    if (wide) return flat_cell(W, s, (int)e);
    return make_int3((int)(e & 1023u), (int)((e >> 10) & 1023u), (int)(e >> 20));
}
#endif

// -------------------------------------------------- mixed batched kernel
// per-thread pair counters
struct PairStats {
    unsigned tets = 0, cand = 0, bbox = 0, in = 0, cin = 0, part = 0, fp64 = 0, fb = 0;
};

// Ill-conditioned tets are listed for route_fp64_kernel: calling their
// (large) routine from the pair loop made the whole loop spill.
__device__ __forceinline__ void route_append(const DepositParams &P, const SharedMixed &S, int tid, int vx, int vy)
{
    const unsigned long long n = atomicAdd(P.route_count, 1ull);
    const int v0 = S.cubes[tid / 6], r = small_div(v0, vx), i = v0 - r * vx, k = small_div(r, vy), j = r - k * vy;
    if (n < P.route_cap)
        P.route[n] = ((unsigned long long)S.item << 16) |
                     (unsigned long long)((i + (vx - 1) * (j + (vy - 1) * k)) * 6 + tid % 6);
    else
        atomicOr(P.error, 4);
}

// Set-up phase: this warp's tets of the wave [first, end) of the tets of the
// item's live cubes.
template <bool kExactD>
__device__ __forceinline__ void wave_setup(const DepositParams &P, SharedMixed &S, const Item &it, int first, int end,
                                           int vx, int vy, int odd, unsigned &n_tets)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slot = threadIdx.x, tid = first + slot;
    int cnt = 0;
    bool route64 = false, wide = false;
    if (tid < end) {
        const int t = tid % 6, v0 = S.cubes[tid / 6];
        const ushort4 off = *reinterpret_cast<const ushort4 *>(S.vert_off[t]);
        ushort4 vid = make_ushort4(v0 + off.x, v0 + off.y, v0 + off.z, v0 + off.w);
        uint2 mn = S.range[vid.x], mx = mn;
        uint32_t flags = mn.y;
        const int more[3] = {vid.y, vid.z, vid.w};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const uint2 w = S.range[more[q]];
            flags |= w.y;
            mn.x = __vminu2(mn.x, w.x);
            mx.x = __vmaxu2(mx.x, w.x);
            mn.y = __vminu2(mn.y, w.y);
            mx.y = __vmaxu2(mx.y, w.y);
        }
        // the orientation rule needs the positions themselves (L1 hits: the block was just staged)
        const int r = small_div(v0, vx), i = v0 - r * vx, k = small_div(r, vy), j = r - k * vy;
        const long long gi = it.base + i + P.stride_y * j + P.stride_z * k;
        const int4 so = *reinterpret_cast<const int4 *>(S.src_off[t]);
        const int sgn = vol6_sign_ref(vol6_exact(load_vertex(P, gi + so.x), load_vertex(P, gi + so.y),
                                                 load_vertex(P, gi + so.z), load_vertex(P, gi + so.w)));
        if (sgn < 0) vid = make_ushort4(vid.w, vid.y, vid.z, vid.x);
        S.wt.vid[slot] = vid;
        // the tet's AABB strictly overlaps the grid box, and its volume is not zero
        if ((flags & (kBelowMax | kAboveMin)) == (kBelowMax | kAboveMin) && sgn != 0)
            cnt = setup_frame<kExactD>(
                mn, mx,
                [&](int q, int a, float &h, float &l) {
                    const int v = q == 0 ? vid.x : (q == 1 ? vid.y : (q == 2 ? vid.z : vid.w));
                    h = S.wt.gh[a][v];
                    l = S.wt.gl[a][v];
                },
                S.g, S.wt, slot, P.error, &route64, &wide);
        if (cnt > 0 && wide) atomicOr(&S.flags[odd], kWideTet);
    }
    n_tets += (cnt > 0);
    if (route64 && cnt > 0) {  // deposited by route_fp64_kernel
        cnt = 0;
        route_append(P, S, tid, vx, vy);
    }
    __syncwarp();
    // exclusive scan of the pair counts across the warp
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const unsigned some = __ballot_sync(0xffffffffu, cnt > 0);
    if (cnt > 0) {
        const int k = 32 * warp + __popc(some & ((1u << lane) - 1));
        S.start[k] = incl - cnt;
        S.tet[k] = (uint8_t)slot;
    }
    if (lane >= __popc(some)) S.start[slot] = INT_MAX;
    if (lane == 31) {
        S.warp_pairs[warp] = incl;
        if (incl > kMaxPartPairs / kWarps) atomicOr(&S.flags[odd], kManyPairs);
    }
}

// The next part of a wave that has kManyPairs, from warp `first` on: the pairs
// of the other warps are set to none.  Returns the part's pairs, 0 after the
// last.  (The whole CTA.)
__device__ __noinline__ int wave_next_part(SharedMixed &S, int first)
{
    if (first == 0) {
        if (threadIdx.x < kWarps) S.all_pairs[threadIdx.x] = S.warp_pairs[threadIdx.x];
        __syncthreads();
    }
    int total;
    const int end = wave_part(S.all_pairs, first, total), w = threadIdx.x;
    __syncthreads();
    if (w < kWarps) S.warp_pairs[w] = w >= first && w < end ? S.all_pairs[w] : 0;
    if (w == 0) {
        S.cursor = 0;
        S.part_end = end;
    }
    __syncthreads();
    return total;
}

// Of 32 pairs, the bit of the one a tet starts at: its start and the pair
// `skip` in the numbering of its warp (start: INT_MAX for none).  0 if it is at
// or before that pair or past the 32.
ADECO_HD inline unsigned start_bit(int start, int rel, int skip)
{
    const unsigned at = (unsigned)start - (unsigned)rel + (unsigned)skip;  // below 2^32: no wrap for a start past rel
    return start > rel && at < 32u ? 1u << at : 0u;
}

// Classify phase: the warps take the wave's candidate pairs 32 at a time and
// classify them; inside cells are deposited at once, partial cells listed, and
// those that one face cuts at the list's end (with the face in the top bits):
// their closed form, for a few lanes of nearly every 32, had taken more than
// the classification itself.  Until no pair is left or the list might not hold
// the 32 pairs each warp may have in hand (`room` of it are used).
// kExactD (zoom grids): whole tets are added where a lane finds them; octree
// leaves of 256^3 take 0.6% longer so, fine zoom grids 3% the other way.
template <bool kStats, bool kExactD>
__device__ __forceinline__ void wave_classify(const DepositParams &P, SharedMixed &S, int *list_n, int *cut_n, int room, bool wide,
                                              PairStats &st)
{
    const int lane = threadIdx.x & 31;
    const unsigned le = 0xffffffffu >> (31 - lane);
    const WaveTets &W = S.wt;
    const GridDesc &g = S.g;
    // lane w: warp w's pairs, and the pairs of the warps before it
    const int own = lane < kWarps ? S.warp_pairs[lane] : 0;
    int pre = own;
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += y;
    }
    const int total = __shfl_sync(0xffffffffu, pre, kWarps - 1);
    pre -= own;
    for (;;) {
        int c0 = 0;
        if (lane == 0)
            c0 = *(volatile int *)list_n + *(volatile int *)cut_n > room - kThreads ? INT_MAX : atomicAdd(&S.cursor, 32);
        c0 = __shfl_sync(0xffffffffu, c0, 0);
        if (c0 >= total) break;
        // The pair's tet, without a search per lane: lane k holds the start of
        // a warp's k-th tet; the last start at or before the first pair, and
        // the starts among the 32 as a bit mask.  Pairs q0.. of one warp's
        // tets at a time: most 32s need one round.
        const int pidx = c0 + lane;
        int s = 0, local = 0;
        for (int q0 = c0;;) {
            const int w = __popc(__ballot_sync(0xffffffffu, lane < kWarps && pre <= q0)) - 1;
            const int before = __shfl_sync(0xffffffffu, pre, w), end = before + __shfl_sync(0xffffffffu, own, w);
            const int start = S.start[32 * w + lane], rel = q0 - before;
            const int first = __popc(__ballot_sync(0xffffffffu, start <= rel)) - 1;
            const unsigned starts = __reduce_or_sync(0xffffffffu, start_bit(start, rel, q0 - c0));
            const int k = first + __popc(starts & le), from = __shfl_sync(0xffffffffu, start, k);
            if (pidx >= q0 && pidx < end) {
                s = S.tet[32 * w + k];
                local = pidx - before - from;
            }
            q0 = end;
            if (q0 >= min(c0 + 32, total)) break;
        }
        bool part = false, holds = false;
        int cross = -1;
        uint32_t entry = 0;
        int3 c = make_int3(0, 0, 0);
        if (pidx < total) {
            c = flat_cell(W, s, local);
            entry = wide ? (uint32_t)local : ((uint32_t)c.x | ((uint32_t)c.y << 10) | ((uint32_t)c.z << 20));
            if (kStats) ++st.cand;
            bool f64 = false;
            const int cls = classify_pair(W, g, s, c.x, c.y, c.z, f64, cross);
            if (kStats) {
                st.fp64 += f64;
                st.in += cls == P_TET_INSIDE;
                st.cin += cls == P_CELL_INSIDE;
                st.part += cls == P_PARTIAL;
                st.bbox += cls != P_NO;
            }
            part = cls == P_PARTIAL && cross < 0;
            holds = cls == P_TET_INSIDE;
            if (kExactD && holds) scatter_whole(P, g, W, s, c.x, c.y, c.z, __activemask());
            const float m = cls == P_CELL_INSIDE ? 6.f * W.f6[s] : 0.f;
            if (m > 0.f) scatter(P, g, W, s, c.x, c.y, c.z, m);
        }
        if (!kExactD) {
            const unsigned lanes = __ballot_sync(0xffffffffu, holds);
            if (holds) scatter_whole(P, g, W, s, c.x, c.y, c.z, lanes);
        }
        const unsigned bal = __ballot_sync(0xffffffffu, part), cut = __ballot_sync(0xffffffffu, cross >= 0);
        const unsigned lt = le >> 1;
        int at = 0;
        if (lane == 0 && bal) at = atomicAdd(list_n, __popc(bal));
        if (lane == 1 && cut) at = atomicAdd(cut_n, __popc(cut));
        const int cut_at = kPairs - 1 - (__shfl_sync(0xffffffffu, at, 1) + __popc(cut & lt));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & lt);
        if (cross >= 0) {
            at = cut_at;
            entry |= (uint32_t)cross << 30;
        }
        if (part || cross >= 0) {
            S.list.cell[at] = entry;
            S.list.tet[at] = (uint8_t)s;
        }
    }
}

// Persistent: CTAs take work items (grid x vertex block) from a global
// counter and deposit an item's tets in waves of kWave (see the top of the
// file).  A wave whose partial pairs do not fit the list is clipped in parts.
// What bounds it is issue (58% of the slots on octree leaves of a 192^3
// lattice, ALU pipe 52% busy, DRAM idle); of the warps' cycles the clipping
// takes 53%, the wait at its end 9, classification 13, set-up 9, staging 6,
// masses 5.  256^3 octree leaves 43.1 ms with a warp in each phase for itself,
// 29.0 now; one 128^3 zoom grid (whole call) 5.3 -> 2.7 ms; a 96^3 grid's
// no-allocation call 4.9 -> 2.3 ms.
// kStats: count the pairs (collect_stats); a separate instantiation, so that
// the others carry no counters.  kExactD: see setup_frame.
template <bool kStats, bool kExactD = false>
__global__ void __launch_bounds__(kThreads, 2) deposit_mixed_kernel(DepositParams P)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SharedMixed &S = *reinterpret_cast<SharedMixed *>(smem_raw);
    const int warp = threadIdx.x >> 5;
    if (P.nothing && *P.nothing) return;
    PairStats st;
    int turn = 0, odd = 0;  // the pair list's counters and the wave's flag in use
    if (threadIdx.x == 0) S.flags[0] = S.list.n[0] = S.list.next[0] = S.cut[0] = S.cut_next[0] = 0;
    const int room = kPairs / kQueue * min(max(P.clip_batch, 64), kQueue);

    for (int taken = 0;; ++taken) {
        // one-item CTAs (serving): a CTA exits after its items, so that the
        // CTAs of other requests' launches get SMs as these finish
        if (P.per_cta_items > 0 && taken >= P.per_cta_items) break;
        if (threadIdx.x == 0) {
            const int unit = atomicAdd(P.counter, 1);
            S.item = unit / P.parts;
            S.part = unit - S.item * P.parts;
            S.n_cubes = 0;
        }
        __syncthreads();
        if (S.item >= P.n_items) break;
        const Item it = P.items[S.item];
        if (threadIdx.x == 0) S.g = P.grids[it.grid];
        const int vx = it.nv & 0xff, vy = (it.nv >> 8) & 0xff, vz = (it.nv >> 16) & 0xff;
        stage_block(P, it, P.grids[it.grid], S, vx, vy, vz);
        __syncthreads();
        const int cvx = vx - 1, cvy = vy - 1, cvz = vz - 1;
        const int ncube = (cvx > 0 && cvy > 0 && cvz > 0) ? cvx * cvy * cvz : 0;
        // the live ones of this CTA's cubes (every parts-th)
        for (int c = S.part + threadIdx.x * P.parts; c < ncube; c += blockDim.x * P.parts) {
            const int r = small_div(c, cvx), k = small_div(r, cvy);
            const int v0 = c - r * cvx + vx * (r - k * cvy + vy * k);
            if (cube_alive(S, v0, vx, vy)) S.cubes[atomicAdd(&S.n_cubes, 1)] = (uint16_t)v0;
        }
        __syncthreads();
        // waves of equal size: a whole meta-cell's 2058 tets are 9 of 229, not
        // 8 of 256 and one of 10
        const int ntet = 6 * S.n_cubes;
        const int nwave = (ntet + kWave - 1) / kWave, wave = nwave ? (ntet + nwave - 1) / nwave : 0;
        for (int first = 0; first < ntet; first += wave) {
            // every warp is through with the wave before
            if (threadIdx.x == 0) S.cursor = S.flags[odd ^ 1] = 0;
            wave_setup<kExactD>(P, S, it, first, min(first + wave, ntet), vx, vy, odd, st.tets);
            __syncthreads();
            const int flags = S.flags[odd];
            const bool wide = (flags & kWideTet) != 0;
            unsigned sum = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) sum += (unsigned)S.warp_pairs[w];
            int total = (flags & kManyPairs) ? wave_next_part(S, 0) : (int)sum;
            bool left = total > 0;
            if (!left) __syncthreads();  // the next wave's set-up writes what this one's warps read above
            while (left) {
                wave_classify<kStats, kExactD>(P, S, &S.list.n[turn], &S.cut[turn], room, wide, st);
                __syncthreads();
                left = S.cursor < total;
                const int np = S.list.n[turn];
                if (threadIdx.x == 0) {  // the next list's
                    S.list.n[turn ^ 1] = 0;
                    S.list.next[turn ^ 1] = 0;
                    S.cut[turn ^ 1] = 0;
                    S.cut_next[turn ^ 1] = 0;
                }
                uint64_t mine = clip_pairs(
                    S.pool[warp], S.list, &S.list.next[turn], np,
                    [&](int j, float *p) {
                        const int s = S.list.tet[j];
                        const int3 c = pair_cell(S.wt, s, S.list.cell[j], wide);
                        piece_coords(S.wt, S.g, s, c.x, c.y, c.z, p);
                    },
                    st.fb);
                // the masses of this warp's pairs
                while (mine) {
                    const int j = 32 * (__ffsll((long long)mine) - 1) + (threadIdx.x & 31);
                    mine &= mine - 1;
                    if (j < np) {
                        const int s = S.list.tet[j];
                        const int3 c = pair_cell(S.wt, s, S.list.cell[j], wide);
                        const long long v = S.list.volume(j);
                        if (v > 0) scatter(P, S.g, S.wt, s, c.x, c.y, c.z, pair_mass(v, S.wt.f6[s]));
                    }
                }
                // one face cuts the cell: closed form, no clipping; taken by the
                // warps that are through with their pairs first
                for (const int ncut = S.cut[turn];;) {
                    int j = 0;
                    if ((threadIdx.x & 31) == 0) j = ncut ? atomicAdd(&S.cut_next[turn], 32) : 0;
                    j = __shfl_sync(0xffffffffu, j, 0);
                    if (j >= ncut) break;
                    j += threadIdx.x & 31;
                    if (j < ncut) {
                        const uint32_t e = S.list.cell[kPairs - 1 - j];
                        const int s = S.list.tet[kPairs - 1 - j];
                        const int3 c = pair_cell(S.wt, s, e & 0x3fffffffu, wide);
                        const float m = halfspace_pair_vol6<false, kExactD>(S.wt, S.g, s, c.x, c.y, c.z, (int)(e >> 30)) * S.wt.f6[s];
                        if (m > 0.f) scatter(P, S.g, S.wt, s, c.x, c.y, c.z, m);
                    }
                    __syncwarp();
                }
                turn ^= 1;
                __syncthreads();
                if (!left && (flags & kManyPairs)) {
                    total = wave_next_part(S, S.part_end);
                    left = total > 0;
                }
            }
            odd ^= 1;
        }
        __syncthreads();
    }
    if (kStats) {
        warp_stat(P.stats, ST_TETS, st.tets);
        warp_stat(P.stats, ST_CAND, st.cand);
        warp_stat(P.stats, ST_BBOX, st.bbox);
        warp_stat(P.stats, ST_INSIDE, st.in);
        warp_stat(P.stats, ST_CELLIN, st.cin);
        warp_stat(P.stats, ST_PARTIAL, st.part);
        warp_stat(P.stats, ST_FP64, st.fp64);
        warp_stat(P.stats, ST_FALLBACK, st.fb);
    }
}

// ------------------------------------------------------ plain FP64 kernel
}  // namespace adeco
#include "plain_fp64.cuh"
#include "route_fp64.cuh"
namespace adeco {

// ------------------------------------------- parity / diagnostics kernels
// Per tet of a patch sequence: vertex slots after the orientation rule, the
// volume sign, in-grid flag and candidate range (13 ints, as the oracle's
// records); and per cell the number of tets whose candidate range covers it.
__global__ void tet_records_kernel(const float *patches, int m, long long cube_begin, long long cube_end,
                                   GridDesc g, int order, int *rec, unsigned int *cand)
{
    const long long cube = cube_begin + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (cube >= cube_end) return;
    const long long cpp = (long long)m * m * m;
    const long long fpp = 3LL * (m + 1) * (m + 1) * (m + 1);
    const float *patch = patches + (cube / cpp) * fpp;
    const int local = (int)(cube % cpp);
    const int k = local / (m * m), r = local % (m * m), j = r / m, i = r % m;
    float3 corner[8];
    for (int s = 0; s < 8; ++s) {
        const int3 o = corner_offset(order, s);
        const long long id = (i + o.x) + (long long)(m + 1) * ((j + o.y) + (long long)(m + 1) * (k + o.z));
        corner[s] = make_float3(patch[3 * id], patch[3 * id + 1], patch[3 * id + 2]);
    }
    for (int t = 0; t < 6; ++t) {
        int *R = rec ? rec + 13 * ((cube - cube_begin) * 6 + t) : nullptr;
        float3 v[4];
        int slot[4];
        for (int q = 0; q < 4; ++q) {
            slot[q] = tet_conn(t, q);
            v[q] = corner[slot[q]];
        }
        const int sgn = vol6_sign_ref(vol6_exact(v[0], v[1], v[2], v[3]));
        if (sgn < 0) { const int tmp = slot[0]; slot[0] = slot[3]; slot[3] = tmp; }
        int lo[3], hi[3];
        const bool in = candidate_range(v, g, lo, hi);
        if (R) {
            for (int q = 0; q < 4; ++q) R[q] = slot[q];
            R[4] = sgn;
            R[5] = in ? 1 : 0;
            for (int a = 0; a < 3; ++a) {
                R[6 + 2 * a] = in ? lo[a] : -1;
                R[7 + 2 * a] = in ? hi[a] : -1;
            }
            R[12] = 0;
        }
        if (cand && in && sgn != 0)
            for (int z = lo[2]; z <= hi[2]; ++z)
                for (int y = lo[1]; y <= hi[1]; ++y)
                    for (int x = lo[0]; x <= hi[0]; ++x)
                        atomicAdd(cand + x + (long long)g.dims * (y + (long long)g.dims * z), 1u);
    }
}

// Bounding box of the vertices of a patch slice (3 floats each), padding
// vertices (all three coordinates 666) left out: per block min xyz, max xyz
// and a NaN flag (7 floats) into part[blockIdx.x * 7 ...].  A cell a tet
// deposits into lies in the tet's candidate range, inside the box of its
// vertices, so the cells outside this box's range receive nothing.
constexpr int kBoxThreads = 256;
__global__ void __launch_bounds__(kBoxThreads) patch_bbox_kernel(const float *pos, long long nvert, float *part)
{
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    float nan = 0.f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvert; i += (long long)gridDim.x * blockDim.x) {
        const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
        if (x == 666.f && y == 666.f && z == 666.f) continue;
        if (x != x || y != y || z != z) nan = 1.f;
        mn[0] = fminf(mn[0], x); mn[1] = fminf(mn[1], y); mn[2] = fminf(mn[2], z);
        mx[0] = fmaxf(mx[0], x); mx[1] = fmaxf(mx[1], y); mx[2] = fmaxf(mx[2], z);
    }
    __shared__ float red[kBoxThreads / 32][7];
    float v[7] = {mn[0], mn[1], mn[2], mx[0], mx[1], mx[2], nan};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const float w = __shfl_down_sync(0xffffffffu, v[q], o);
            v[q] = (q < 3) ? fminf(v[q], w) : fmaxf(v[q], w);
        }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int q = 0; q < 7; ++q) red[warp][q] = v[q];
    __syncthreads();
    if (threadIdx.x < 7) {
        const int q = threadIdx.x;
        float r = red[0][q];
        for (int w = 1; w < kBoxThreads / 32; ++w) r = (q < 3) ? fminf(r, red[w][q]) : fmaxf(r, red[w][q]);
        part[blockIdx.x * 7 + q] = r;
    }
}

// The vertices' box over all passes of a call, and its cell range.
struct CallBox {
    float vmin[3], vmax[3];
    int nan;
    int empty;           // no cell of the grid can have received mass
    int lo[3], ext[3];   // the cells that can
};

// Starts a boundary call's pass, one launch instead of three copies and three
// clears: work items of patches [p0, p0 + np) of (m + 1)^3 vertices (sub-blocks
// of at most 7^3 cubes, nsb per axis), their cubes' offsets (cube_off, for the
// FP64 path, or null), the grid descriptor, and zeroed counters.  first: the
// call's first pass, which also clears the error flag and the box.
__global__ void patch_items_kernel(Item *items, long long *cube_off, long long p0, int n_items, int m, int nsb,
                                   GridDesc *grid, GridDesc g, int *counter, unsigned long long *route_count, CallBox *box,
                                   int first)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        *grid = g;
        counter[0] = 0;
        if (first) counter[1] = 0;
        if (route_count) *route_count = 0;
        if (box && first) {
            for (int a = 0; a < 3; ++a) {
                box->vmin[a] = INFINITY;
                box->vmax[a] = -INFINITY;
            }
            box->nan = 0;
        }
    }
    if (i >= n_items) return;
    const long long n1 = m + 1, n2 = n1 * n1;
    const int per = nsb * nsb * nsb;
    const long long p = i / per;
    const int sb = i % per, sx = sb % nsb, sy = (sb / nsb) % nsb, sz = sb / (nsb * nsb);
    const int ox = sx * 7, oy = sy * 7, oz = sz * 7;
    const int vx = min(8, m + 1 - ox), vy = min(8, m + 1 - oy), vz = min(8, m + 1 - oz);
    Item it;
    it.base = (p0 + p) * n1 * n2 + ox + n1 * oy + n2 * oz;
    it.grid = 0;
    it.nv = vx | (vy << 8) | (vz << 16);
    items[i] = it;
    if (cube_off) {
        // whole slabs, then whole rows of this slab, then blocks of this row
        const long long before = p * m * m * m + (long long)oz * m * m + (long long)(vz - 1) * ((long long)oy * m + (long long)(vy - 1) * ox);
        cube_off[i] = before;
    }
}

// Adds a pass's block boxes (patch_bbox_kernel) to the call's box and forms its
// cell range: one cell of margin against the rounding of the kernels' FP32
// range arithmetic; a NaN coordinate takes the whole grid.  host: a copy for the
// host, in page-locked memory, or null.
__global__ void __launch_bounds__(7 * 32) call_box_kernel(const float *part, int nblocks, const GridDesc *gp, CallBox *box,
                                                          CallBox *host)
{
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;  // a warp per number of the box, the last for the NaN flag
    float r = q < 3 ? INFINITY : (q < 6 ? -INFINITY : 0.f);
    for (int b = lane; b < nblocks; b += 32) r = q < 3 ? fminf(r, part[7 * b + q]) : fmaxf(r, part[7 * b + q]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float w = __shfl_xor_sync(0xffffffffu, r, o);
        r = q < 3 ? fminf(r, w) : fmaxf(r, w);
    }
    if (lane == 0) {
        if (q < 3) box->vmin[q] = fminf(box->vmin[q], r);
        else if (q < 6) box->vmax[q - 3] = fmaxf(box->vmax[q - 3], r);
        else if (r != 0.f) box->nan = 1;
    }
    __syncthreads();
    if (q) return;  // a lane per axis
    const GridDesc &g = *gp;
    const int a = lane;
    bool empty = false;
    if (a < 3) {
        int lo = 0, ext = g.dims;
        if (!box->nan) {
            const double gmin = g.gmin[a], gmax = g.gmax[a], delta = g.delta[a];
            const float vmin = box->vmin[a], vmax = box->vmax[a];
            if (!(vmin <= vmax) || (double)vmax < gmin || (double)vmin > gmax || !(delta > 0.0)) {
                empty = true;
            } else {
                const double flo = floor((fmax((double)vmin, gmin) - gmin) / delta) - 1.0;
                const double fhi = ceil((fmin((double)vmax, gmax) - gmin) / delta) + 1.0;
                const int l = (int)fmin(fmax(flo, 0.0), (double)(g.dims - 1)), h = (int)fmin(fmax(fhi, 0.0), (double)(g.dims - 1));
                lo = l;
                ext = h - l + 1;
            }
        }
        box->lo[a] = lo;
        box->ext[a] = ext;
    }
    empty = __any_sync(0xffffffffu, empty);
    if (lane == 0) box->empty = empty;
    __syncwarp();  // the lanes' axes are written
    if (lane == 0 && host) *host = *box;
}

// A pass's sums of the box's cells, from the fixed point grid (times scale)
// when `fixed` is set, else from `f64`.
__device__ __forceinline__ double box_value(const unsigned long long *fixed, const double *f64, long long c, double scale)
{
    return fixed ? (double)fixed[c] * scale : f64[c];
}

// The box's cells, packed x fastest, for a host that adds them itself.
__global__ void grid_box_kernel(const unsigned long long *fixed, const double *f64, double *out, int dims, int lo0,
                                int lo1, int lo2, int e0, int e1, int e2, double scale)
{
    const long long n = (long long)e0 * e1 * e2;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / e0;
        const int x = (int)(i - r * e0), y = (int)(r % e1), z = (int)(r / e1);
        out[i] = box_value(fixed, f64, (lo0 + x) + (long long)dims * ((lo1 + y) + (long long)dims * (lo2 + z)), scale);
    }
}

// The same cells added into the caller's grid in host memory, where the device
// reads and writes pageable memory through the host's page tables: 128^3 cells
// 62 us against 530 us for the copy's additions on a host core.  Adds nothing
// if the call failed.
template <typename T>
__global__ void host_accumulate_kernel(const unsigned long long *fixed, const double *f64, T *out, int dims,
                                       const CallBox *box, const int *error, double scale)
{
    if (*error || box->empty) return;
    const int e0 = box->ext[0], e1 = box->ext[1];
    const long long n = (long long)e0 * e1 * box->ext[2];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / e0;
        const int x = (int)(i - r * e0), y = (int)(r % e1), z = (int)(r / e1);
        const long long c = (box->lo[0] + x) + (long long)dims * ((box->lo[1] + y) + (long long)dims * (box->lo[2] + z));
        out[c] += (T)box_value(fixed, f64, c, scale);
    }
}

// fixed-point sums -> FP64 masses, added into an FP64 grid unless the call failed
__global__ void fixed_accumulate_f64_kernel(const unsigned long long *in, double *out, long long n, double scale,
                                            const int *error)
{
    if (*error) return;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] += (double)in[i] * scale;
}

// per-leaf fixed-point grids -> FP64 with each grid's own scale
__global__ void fixed_to_f64_grids_kernel(const unsigned long long *in, double *out, const GridDesc *grids,
                                          int n_grids, long long cells_per_grid)
{
    const long long n = (long long)n_grids * cells_per_grid;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int gi = (int)(i / cells_per_grid);
        out[i] = ldexp((double)in[i], -grids[gi].shift);
    }
}

// Meta-cell AABBs of a resident float4 lattice (7^3-cube meta-cells): one
// warp per meta-cell, min/max over its <= 8^3 vertices.
__global__ void meta_bbox_kernel(const float4 *pos, int nx, int ny, int nz, int cdx, int cdy, int cdz, float *bbox6)
{
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long nmc = (long long)cdx * cdy * cdz;
    if (w >= nmc) return;
    const int cx = (int)(w % cdx), r = (int)(w / cdx), cy = r % cdy, cz = r / cdy;
    const int ox = cx * 7, oy = cy * 7, oz = cz * 7;
    const int dx = (cx + 1 == cdx) ? nx - ox : 8, dy = (cy + 1 == cdy) ? ny - oy : 8, dz = (cz + 1 == cdz) ? nz - oz : 8;
    float mn[3] = {3.4e38f, 3.4e38f, 3.4e38f}, mx[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    const int nv = dx * dy * dz;
    for (int v = lane; v < nv; v += 32) {
        const int i = v % dx, rr = v / dx, j = rr % dy, k = rr / dy;
        const float4 p = pos[(ox + i) + (long long)nx * ((oy + j) + (long long)ny * (oz + k))];
        mn[0] = fminf(mn[0], p.x); mx[0] = fmaxf(mx[0], p.x);
        mn[1] = fminf(mn[1], p.y); mx[1] = fmaxf(mx[1], p.y);
        mn[2] = fminf(mn[2], p.z); mx[2] = fmaxf(mx[2], p.z);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            mn[a] = fminf(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
            mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
        }
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            bbox6[6 * w + a] = mn[a];
            bbox6[6 * w + 3 + a] = mx[a];
        }
}

}  // namespace adeco

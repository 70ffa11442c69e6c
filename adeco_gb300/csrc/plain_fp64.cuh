// plain_fp64.cuh -- the plain FP64 deposit: every tet set up, classified and
// clipped in FP64, masses added with FP64 atomics, one launch per request.
// The precision the batched kernel is measured against, and the boundary's
// ADECO_PREC_FP64.  Included by kernels.cuh.
//
// A warp takes 5 lattice cubes (30 tets, a lane each) through set-up,
// classification and clipping.  The candidate cells of the 30 tets are
// flattened across the lanes, partial cells are listed and clipped by the
// whole warp, a lane per piece, with the steps of the mixed path's engine
// (clip_engine.cuh) on FP64 pieces.  A lane per cell with a local-memory
// stack, one tet of a cube at a time, had left most lanes idle and every
// piece in local memory: 24^3 cubes onto 40^3 cells 88 ms, now 3.8 ms.  What
// bounds it is the FP64 pipe (70% of cycles busy; one warp instruction takes
// it about 15 cycles), so face tests and clamps are integer compares of the
// bits, and a quotient is a product with a Newton step's reciprocal, corrected
// by its remainder (4.45 -> 3.8 ms).
#pragma once

namespace adeco {

constexpr int kPlainThreads = 128;
constexpr int kPlainWarps = kPlainThreads / 32;
constexpr int kPlainCubes = 5;   // most cubes a warp takes together (30 tets, a lane each)
constexpr int kPlainPool = 64;   // pieces per warp pool
constexpr int kPlainRoom = kPlainPool - 8;  // what steps of several lanes may fill (see plain_clip)
constexpr int kPlainLast = 64;   // pieces at their last crossed face per warp
constexpr int kPlainList = 128;  // partial cells per warp list

struct PlainWarp {
    // the tets, in their anchor cells' frames
    double q[4][3][32];   // vertices
    double n[4][3][32];   // inward face normals, inside <=> n.x - d > 0
    double d[4][32];
    double pp[4][32], pm[4][32];  // sums of a normal's positive / negative parts
    double bmin[3][32], bmax[3][32];
    double f6[32];        // mass per unit of 6x clipped volume
    long long scan[33];   // work units (cells, or rows of 8 or more cells) of the tets before this one
    int lo[3][32], ex[3][32];
    // clipping
    double v[12][kPlainPool];
    uint32_t flags[kPlainPool];
    uint32_t owner[kPlainPool];
    double last[5][kPlainLast];
    uint32_t last_meta[kPlainLast];  // inside mask | upper face << 4 | owner << 8
    unsigned long long cell[kPlainList];  // a | b << 13 | c << 26 | tet << 39
    double vol[kPlainList];               // 6x volume of each listed cell
};
constexpr size_t kPlainSmem = sizeof(PlainWarp) * kPlainWarps;

// The inside flags of a point as face_bits, from the bits of its coordinates.
__device__ __forceinline__ int face_bits_f64(const double x[3])
{
    int b = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const long long u = __double_as_longlong(x[a]);
        b |= ((u > 0) ? 1 : 0) << (2 * a);                                      // x > 0
        b |= (((int)(u >> 32) < 0x3ff00000) ? 1 : 0) << (2 * a + 1);           // x < 1
    }
    return b;
}

// x limited to [0, 1], by its bits
__device__ __forceinline__ double sat01_f64(double x)
{
    const int hi = __double2hiint(x);
    return hi < 0 ? 0.0 : (hi >= 0x3ff00000 ? 1.0 : x);
}

// 1 / d to about 38 bits from an approximation r of 19 or more: one step of
// Newton's iteration.
ADECO_HD inline double rcp_f64(double d, double r) { return fma(r, fma(-d, r, 1.0), r); }

// num / d to half an ulp, given r = rcp_f64(d): the product num r corrected by
// its remainder, which squares the error of r (Markstein 1990).  A second
// Newton step instead of the correction left errors of up to 1.4 ulp.
ADECO_HD inline double quot_f64(double num, double d, double r)
{
    const double q = num * r;
    return fma(fma(-d, q, num), r, q);
}

// rcp_f64 from the hardware's approximation (PTX rcp.approx.ftz.f64), for a
// difference of cell-frame coordinates across a face: nonzero and far from the
// range limits.
__device__ __forceinline__ double face_rcp(double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    return rcp_f64(d, r);
}

__device__ __forceinline__ double sel4_f64(int i, double a, double b, double c, double d)
{
    return (i & 2) ? ((i & 1) ? d : c) : ((i & 1) ? b : a);
}

// side_fraction (clip_engine.cuh) in FP64
__device__ __forceinline__ double side_fraction_f64(double x0, double x1, double x2, double x3, int mask, double plane)
{
    const int pm = split_perm(mask), k = split_kin(mask);
    const bool k1 = k == 1, k2 = k == 2, k3 = k == 3;
    const double a = sel4_f64(pm & 3, x0, x1, x2, x3), b = sel4_f64((pm >> 2) & 3, x0, x1, x2, x3);
    const double c = sel4_f64((pm >> 4) & 3, x0, x1, x2, x3), d = sel4_f64((pm >> 6) & 3, x0, x1, x2, x3);
    const double in[4] = {a, k3 ? b : a, k1 ? a : (k2 ? b : c), b};
    const double out[4] = {k1 ? b : (k2 ? c : d), k1 ? c : d, k2 ? c : d, d};
    double t[4], w[4] = {1.0, 1.0, 1.0, 1.0}, r[4] = {1.0, 1.0, 1.0, 1.0};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (e == 3 && !k2) {  // only two inside vertices have a fourth edge
            t[e] = 0.0;
            continue;
        }
        w[e] = out[e] - in[e];
        r[e] = face_rcp(w[e]);
        t[e] = sat01_f64(quot_f64(plane - in[e], w[e], r[e]));
    }
    if (k1) return t[0] * t[1] * t[2];
    // u = 1 - t of the edges that have one: BC and BD (two inside), AD and BD (three)
    const double ua = sat01_f64(quot_f64((k2 ? out[2] : out[0]) - plane, k2 ? w[2] : w[0], k2 ? r[2] : r[0]));
    const double ub = sat01_f64(quot_f64((k2 ? out[3] : out[1]) - plane, k2 ? w[3] : w[1], k2 ? r[3] : r[1]));
    if (k2) return fma(t[2], t[3], t[0] * (t[3] * ua + t[1] * ub));
    return fma(ua, fma(ub, t[2], t[1]), t[0]);
}

__device__ __forceinline__ void plain_put_last(PlainWarp &W, int slot, const double p[12], int f, int mask, int owner)
{
    const int axis = f >> 1;
    W.last[0][slot] = fabs(vol6_fast<double>(p, p + 3, p + 6, p + 9));
#pragma unroll
    for (int q = 0; q < 4; ++q) W.last[1 + q][slot] = axis == 0 ? p[3 * q] : (axis == 1 ? p[3 * q + 1] : p[3 * q + 2]);
    W.last_meta[slot] = (uint32_t)(mask | ((f & 1) << 4) | (owner << 8));
}

// The warp's listed cells, clipped: W.vol[j] of j < np are their 6x volumes.
// Steps and their order as clip_pairs.
__device__ __forceinline__ void plain_clip(PlainWarp &W, const GridDesc &g, int np)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1;
    int top = 0, nlast = 0, next = 0;
    for (;;) {
        if (nlast >= 32 || (nlast && !top && next >= np)) {
            const int n = min(nlast, 32), idx = nlast - 1 - lane;
            if (lane < n) {
                const uint32_t m = W.last_meta[idx];
                const double frac = side_fraction_f64(W.last[1][idx], W.last[2][idx], W.last[3][idx], W.last[4][idx],
                                                      m & 15, (m & 16) ? 1.0 : 0.0);
                atomicAdd(&W.vol[m >> 8], W.last[0][idx] * frac);
            }
            nlast -= n;
            __syncwarp();
            continue;
        }
        if (top < 32 && next < np) {
            const int nb = min(min(32, np - next), min(kPlainRoom - top, kPlainLast - nlast)), j = next + lane;
            bool push = false, last = false;
            double p[12];
            uint32_t flags = 0;
            int f = 0, mask = 0;
            if (lane < nb) {
                const unsigned long long e = W.cell[j];
                const int s = (int)(e >> 39);
                const int c[3] = {(int)(e & 8191u), (int)((e >> 13) & 8191u), (int)((e >> 26) & 8191u)};
                int b[4];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const double o = c[x] * g.rcell[x];
#pragma unroll
                    for (int q = 0; q < 4; ++q) p[3 * q + x] = W.q[q][x][s] - o;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) b[q] = face_bits_f64(p + 3 * q);
                flags = (uint32_t)(b[0] | (b[1] << 6) | (b[2] << 12) | (b[3] << 18));
                const int code = next_face(b[0], b[1], b[2], b[3], 0, f, mask, last);
                push = code == 2 && !last;
                last = code == 2 && last;
                W.vol[j] = code == 1 ? fabs(vol6_fast<double>(p, p + 3, p + 6, p + 9)) : 0.0;
            }
            const unsigned pushing = __ballot_sync(0xffffffffu, push), lasts = __ballot_sync(0xffffffffu, last);
            if (push) {
                const int slot = top + __popc(pushing & lt);
#pragma unroll
                for (int x = 0; x < 12; ++x) W.v[x][slot] = p[x];
                W.flags[slot] = flags;
                W.owner[slot] = (uint32_t)j;
            }
            if (last) plain_put_last(W, nlast + __popc(lasts & lt), p, f, mask, j);
            top += __popc(pushing);
            nlast += __popc(lasts);
            next += nb;
            __syncwarp();
            continue;
        }
        if (!top) break;
        const int n = min(top, 32), idx = top - 1 - lane;  // split step: lane l takes slot top - 1 - l
        int owner = 0;
        int code[3] = {0, 0, 0};
        uint32_t cflags[3] = {0, 0, 0};
        int cface[3], cmask[3];
        double A[3], B[3], C[3], E[4][3];
        bool k1 = false, k2 = false;
        if (lane < n) {
            const uint32_t m = W.flags[idx];
            owner = (int)W.owner[idx];
            const int done = 63 & ~(int)(m | (m >> 6) | (m >> 12) | (m >> 18));
            int f, mask;
            bool last;
            next_face(m & 63, (m >> 6) & 63, (m >> 12) & 63, (m >> 18) & 63, done, f, mask, last);
            const int pm = split_perm(mask), k = split_kin(mask), axis = f >> 1;
            const int ia = pm & 3, ib = (pm >> 2) & 3, ic = (pm >> 4) & 3, id = (pm >> 6) & 3;
            const double plane = (f & 1) ? 1.0 : 0.0;
            k1 = k == 1;
            k2 = k == 2;
            double D[3];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                A[x] = W.v[3 * ia + x][idx];
                B[x] = W.v[3 * ib + x][idx];
                C[x] = W.v[3 * ic + x][idx];
                D[x] = W.v[3 * id + x][idx];
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                double in[3], out[3];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    in[x] = e == 0 ? A[x] : (e == 1 ? (k == 3 ? B[x] : A[x]) : (e == 2 ? (k1 ? A[x] : (k2 ? B[x] : C[x])) : B[x]));
                    out[x] = e == 0 ? (k1 ? B[x] : (k2 ? C[x] : D[x])) : (e == 1 ? (k1 ? C[x] : D[x])
                                                                                  : (e == 2 ? (k2 ? C[x] : D[x]) : D[x]));
                }
                if (e == 3 && !k2) {
                    E[e][0] = E[e][1] = E[e][2] = 0.0;  // not used
                    continue;
                }
                const double din = axis == 0 ? in[0] : (axis == 1 ? in[1] : in[2]);
                const double dout = axis == 0 ? out[0] : (axis == 1 ? out[1] : out[2]);
                const double d = dout - din, t = sat01_f64(quot_f64(plane - din, d, face_rcp(d)));
#pragma unroll
                for (int x = 0; x < 3; ++x) E[e][x] = x == axis ? plane : fma(t, out[x] - in[x], in[x]);
            }
            const int keep = 63 & ~(done | (1 << f));
            const int bA = (int)(m >> (6 * ia)) & keep, bB = (int)(m >> (6 * ib)) & keep, bC = (int)(m >> (6 * ic)) & keep;
            int bE[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) bE[e] = face_bits_f64(E[e]) & keep;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int b1 = c == 0 ? (k1 ? bE[0] : bB) : (c == 1 ? (k2 ? bE[2] : bB) : (k2 ? bE[0] : bE[1]));
                const int b2 = c == 0 ? (k1 ? bE[1] : (k2 ? bE[2] : bC)) : (c == 1 ? (k2 ? bE[0] : bE[2]) : (k2 ? bE[1] : bE[2]));
                const int b3 = c == 0 ? (k2 ? bE[3] : bE[2]) : (c == 1 ? (k2 ? bE[3] : bE[1]) : (k2 ? bE[3] : bE[0]));
                cflags[c] = (uint32_t)(bA | (b1 << 6) | (b2 << 12) | (b3 << 18));
                bool cl;
                code[c] = next_face(bA, b1, b2, b3, 63 & ~keep, cface[c], cmask[c], cl);
                if (code[c] == 2 && !cl) code[c] = 3;
                if (c > 0 && k1) code[c] = 0;
            }
        }
        // When the children do not all fit, the first lanes for which they do
        // commit their step; the pieces of the others, the lower slots, stay
        // where they are.  Lane 0's always fit: steps of several lanes leave 8
        // slots free, and a piece that crosses c faces leaves at most two more
        // pieces in the pool than it took, and only for c = 6, 5, 4 and 3 on
        // the way down (its children cross fewer faces).
        int s_incl = 0, l_incl = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            s_incl += __popc(__ballot_sync(0xffffffffu, code[c] == 3) & (lt << 1 | 1));
            l_incl += __popc(__ballot_sync(0xffffffffu, code[c] == 2) & (lt << 1 | 1));
        }
        const unsigned bad = __ballot_sync(0xffffffffu, lane > 0 && lane < n && (top - (lane + 1) + s_incl > kPlainRoom ||
                                                                               nlast + l_incl > kPlainLast));
        const int commit = bad ? __ffs(bad) - 1 : n;
        if (lane >= commit) code[0] = code[1] = code[2] = 0;
        top -= commit;
        __syncwarp();  // every lane has read its slot
        double v = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const unsigned sm = __ballot_sync(0xffffffffu, code[c] == 3), lm = __ballot_sync(0xffffffffu, code[c] == 2);
            if (code[c]) {
                double ch[12];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    ch[x] = A[x];
                    ch[3 + x] = c == 0 ? (k1 ? E[0][x] : B[x]) : (c == 1 ? (k2 ? E[2][x] : B[x]) : (k2 ? E[0][x] : E[1][x]));
                    ch[6 + x] = c == 0 ? (k1 ? E[1][x] : (k2 ? E[2][x] : C[x]))
                                       : (c == 1 ? (k2 ? E[0][x] : E[2][x]) : (k2 ? E[1][x] : E[2][x]));
                    ch[9 + x] = c == 0 ? (k2 ? E[3][x] : E[2][x]) : (c == 1 ? (k2 ? E[3][x] : E[1][x]) : (k2 ? E[3][x] : E[0][x]));
                }
                if (code[c] == 3) {
                    const int slot = top + __popc(sm & lt);
#pragma unroll
                    for (int x = 0; x < 12; ++x) W.v[x][slot] = ch[x];
                    W.flags[slot] = cflags[c];
                    W.owner[slot] = (uint32_t)owner;
                } else if (code[c] == 2) {
                    plain_put_last(W, nlast + __popc(lm & lt), ch, cface[c], cmask[c], owner);
                } else {
                    v += fabs(vol6_fast<double>(ch, ch + 3, ch + 6, ch + 9));
                }
            }
            top += __popc(sm);
            nlast += __popc(lm);
        }
        if (v > 0.0) atomicAdd(&W.vol[owner], v);
        __syncwarp();
    }
}

// item_cube_offset: the offsets of the items' cubes; the launch
// deposits cubes [cube_begin, cube_end), warp_cubes (at most kPlainCubes) a
// warp at a time.  All items have the same grid.
__global__ void __launch_bounds__(kPlainThreads) deposit_plain_fp64_kernel(DepositParams P, long long cube_begin,
                                                                           long long cube_end,
                                                                           const long long *item_cube_offset,
                                                                           int warp_cubes)
{
    if (P.nothing && *P.nothing) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlainWarp &W = reinterpret_cast<PlainWarp *>(smem_raw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const GridDesc &g = P.grids[P.items[0].grid];
    for (long long base = cube_begin + gw * warp_cubes; base < cube_end; base += nw * warp_cubes) {
        const int sub = lane / 6, t = lane - 6 * sub;
        const long long cube = base + sub;
        long long units = 0;
        bool have = sub < warp_cubes && cube < cube_end, pad = false;
        float3 v[4];
        if (have) {
            // item owning this cube (binary search over the cube offsets)
            int lo_i = 0, hi_i = P.n_items - 1;
            while (lo_i < hi_i) {
                const int mid = (lo_i + hi_i + 1) >> 1;
                if (item_cube_offset[mid] <= cube) lo_i = mid; else hi_i = mid - 1;
            }
            const Item it = P.items[lo_i];
            const int cvx = (it.nv & 0xff) - 1, cvy = ((it.nv >> 8) & 0xff) - 1;
            const int c = (int)(cube - item_cube_offset[lo_i]);
            const int ci = c % cvx, r = c / cvx, cj = r % cvy, ck = r / cvy;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int3 o = corner_offset(P.order, tet_conn(t, q));
                v[q] = load_vertex(P, it.base + (ci + o.x) + P.stride_y * (cj + o.y) + P.stride_z * (ck + o.z));
                if (P.pad_check && P.src_kind != SRC_LATTICE_F4) {
                    const float sum = __fadd_rn(__fadd_rn(fabsf(__fsub_rn(v[q].x, 666.f)), fabsf(__fsub_rn(v[q].y, 666.f))),
                                                fabsf(__fsub_rn(v[q].z, 666.f)));
                    pad |= ((double)sum < 1.E-03);
                }
            }
        }
        // a padding vertex takes all six tets of its cube (which use all eight corners)
        const unsigned pads = __ballot_sync(0xffffffffu, pad);
        have = have && !((pads >> (6 * sub)) & 63u);
        if (have) {
            const int sgn = vol6_sign_ref(vol6_exact(v[0], v[1], v[2], v[3]));
            int lo[3], hi[3];
            if (candidate_range(v, g, lo, hi) && sgn != 0 && tile_clamp(g, lo, hi)) {
                if (sgn < 0) {
                    const float3 tmp = v[0];
                    v[0] = v[3];
                    v[3] = tmp;
                }
                double qd[4][3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const double anchor = fma((double)lo[a], g.delta_d[a], g.gmin_d[a]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const double x = (a == 0) ? (double)v[q].x : ((a == 1) ? (double)v[q].y : (double)v[q].z);
                        qd[q][a] = (x - anchor) * g.scale_d[a];
                        W.q[q][a][lane] = qd[q][a];
                    }
                    W.bmin[a][lane] = fmin(fmin(qd[0][a], qd[1][a]), fmin(qd[2][a], qd[3][a]));
                    W.bmax[a][lane] = fmax(fmax(qd[0][a], qd[1][a]), fmax(qd[2][a], qd[3][a]));
                    W.lo[a][lane] = lo[a];
                    W.ex[a][lane] = hi[a] - lo[a] + 1;
                }
                W.f6[lane] = g.mass_factor / fabs(vol6_fast<double>(qd[0], qd[1], qd[2], qd[3]));
                // inward face planes: faces (0,2,1) (0,3,2) (0,1,3) (1,2,3)
                const int fa[4] = {0, 0, 0, 1}, fb[4] = {2, 3, 1, 2}, fc[4] = {1, 2, 3, 3};
#pragma unroll
                for (int f = 0; f < 4; ++f) {
                    const double e1x = qd[fb[f]][0] - qd[fa[f]][0], e1y = qd[fb[f]][1] - qd[fa[f]][1],
                                 e1z = qd[fb[f]][2] - qd[fa[f]][2];
                    const double e2x = qd[fc[f]][0] - qd[fa[f]][0], e2y = qd[fc[f]][1] - qd[fa[f]][1],
                                 e2z = qd[fc[f]][2] - qd[fa[f]][2];
                    const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
                    W.n[f][0][lane] = nx;
                    W.n[f][1][lane] = ny;
                    W.n[f][2][lane] = nz;
                    W.d[f][lane] = nx * qd[fa[f]][0] + ny * qd[fa[f]][1] + nz * qd[fa[f]][2];
                    W.pp[f][lane] = fmax(nx, 0.0) + fmax(ny, 0.0) + fmax(nz, 0.0);
                    W.pm[f][lane] = fmin(nx, 0.0) + fmin(ny, 0.0) + fmin(nz, 0.0);
                }
                const long long rows = (long long)(hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1);
                const int ex0 = hi[0] - lo[0] + 1;
                units = ex0 < 8 ? rows * ex0 : rows;
            }
        }
        long long incl = units;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        W.scan[lane] = incl - units;
        const long long total = __shfl_sync(0xffffffffu, incl, 31);
        __syncwarp();

        auto put = [&](int s, int a, int b, int c, double m) {
            atomicAdd(P.out_d + g.out_offset + (W.lo[0][s] + a) +
                          (long long)g.dims * ((W.lo[1][s] + b) + (long long)g.dims * (W.lo[2][s] + c)), m);
        };
        int np = 0;  // listed partial cells
        auto flush = [&]() {
            plain_clip(W, g, np);
            __syncwarp();
            for (int j = lane; j < np; j += 32) {
                const unsigned long long e = W.cell[j];
                const int s = (int)(e >> 39);
                const double m = W.vol[j] * W.f6[s];
                if (m > 0.0) put(s, (int)(e & 8191u), (int)((e >> 13) & 8191u), (int)((e >> 26) & 8191u), m);
            }
            np = 0;
            __syncwarp();
        };
        // Work units 32 at a time: a cell, or a row of 8 or more cells along x.
        // The plane bounds are linear in a row's cell index, so each plane
        // bounds it; widened / narrowed by a cell against rounding, cells
        // outside [a, a3] cannot meet the tet and cells of [a1, a2) lie inside
        // it; only the cells in between are tested one by one.
        for (long long u0 = 0; u0 < total; u0 += 32) {
            const long long u = u0 + lane;
            int s = 0, a = 0, a1 = 0, a2 = 0, a3 = -1, b = 0, c = 0;  // cells to test: [a, a1), then [a2, a3]
            if (u < total) {
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (W.scan[s + step] <= u) s += step;
                const int ex0 = W.ex[0][s], ex1 = W.ex[1][s];
                unsigned r = (unsigned)(u - W.scan[s]);  // at most 4096^2 rows, or 7 * 4096^2 cells
                if (ex0 < 8) {
                    a = (int)(r % (unsigned)ex0);
                    a1 = a + 1;
                    r /= (unsigned)ex0;
                    b = (int)(r % (unsigned)ex1);
                    c = (int)(r / (unsigned)ex1);
                } else {
                    b = (int)(r % (unsigned)ex1);
                    c = (int)(r / (unsigned)ex1);
                    const double ob = b * g.rcell[1], oc = c * g.rcell[2];
                    double c0 = 0.0, c1 = ex0 - 1, i0 = 0.0, i1 = ex0 - 1;
                    bool none = false, no_in = false;
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        const double nx = W.n[f][0][s] * g.rcell[0];
                        const double K = W.n[f][1][s] * ob + W.n[f][2][s] * oc - W.d[f][s];
                        if (nx > 0.0) {
                            c0 = fmax(c0, floor(-(K + W.pp[f][s]) / nx) - 1.0);
                            i0 = fmax(i0, floor(-(K + W.pm[f][s]) / nx) + 2.0);
                        } else if (nx < 0.0) {
                            c1 = fmin(c1, ceil(-(K + W.pp[f][s]) / nx) + 1.0);
                            i1 = fmin(i1, ceil(-(K + W.pm[f][s]) / nx) - 2.0);
                        } else {
                            none = none || !(K + W.pp[f][s] > 0.0);
                            no_in = no_in || !(K + W.pm[f][s] > 0.0);
                        }
                    }
                    if (!none) {
                        const int lc = (int)fmax(c0, 0.0), hc = (int)fmin(c1, (double)(ex0 - 1));
                        int li = (int)fmax(i0, (double)lc), hi_ = (int)fmin(i1, (double)hc);
                        if (no_in || li > hi_) {
                            li = hc + 1;
                            hi_ = hc;
                        }
                        for (int x = li; x <= hi_; ++x) put(s, x, b, c, 6.0 * W.f6[s]);
                        a = lc;
                        a1 = li;
                        a2 = hi_ + 1;
                        a3 = hc;
                    }
                }
            }
            for (;;) {
                const bool one = a < a1 || a2 <= a3;
                if (!__any_sync(0xffffffffu, one)) break;
                bool part = false;
                int x = 0;
                if (one) {
                    x = a < a1 ? a++ : a2++;
                    // cell origin in the anchor frame (the cell extends 1 along each axis)
                    const double oa = x * g.rcell[0], ob = b * g.rcell[1], oc = c * g.rcell[2];
                    if (W.bmin[0][s] < oa + 1.0 && oa < W.bmax[0][s] && W.bmin[1][s] < ob + 1.0 && ob < W.bmax[1][s] &&
                        W.bmin[2][s] < oc + 1.0 && oc < W.bmax[2][s]) {
                        bool outside = false, all_in = true;
#pragma unroll
                        for (int f = 0; f < 4; ++f) {
                            const double at = W.n[f][0][s] * oa + W.n[f][1][s] * ob + W.n[f][2][s] * oc - W.d[f][s];
                            if (at + W.pp[f][s] <= 0.0) outside = true;
                            if (!(at + W.pm[f][s] > 0.0)) all_in = false;
                        }
                        if (!outside) {
                            if (W.bmin[0][s] >= oa && W.bmax[0][s] <= oa + 1.0 && W.bmin[1][s] >= ob &&
                                W.bmax[1][s] <= ob + 1.0 && W.bmin[2][s] >= oc && W.bmax[2][s] <= oc + 1.0)
                                put(s, x, b, c, (double)g.tet_mass);
                            else if (all_in)
                                put(s, x, b, c, 6.0 * W.f6[s]);
                            else
                                part = true;
                        }
                    }
                }
                const unsigned bal = __ballot_sync(0xffffffffu, part);
                if (part)
                    W.cell[np + __popc(bal & lt)] = (unsigned long long)x | ((unsigned long long)b << 13) |
                                                    ((unsigned long long)c << 26) | ((unsigned long long)s << 39);
                np += __popc(bal);
                __syncwarp();
                if (np > kPlainList - 32) flush();
            }
        }
        if (np) flush();
    }
}

}  // namespace adeco

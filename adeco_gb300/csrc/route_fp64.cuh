// route_fp64.cuh -- ill-conditioned tets (condition number beyond kKappaFp64),
// listed by deposit_mixed_kernel and deposited by a launch of their own: cells
// classified by FP32 planes and, where those are unsure, FP64 ones; shares of
// the tet from barycentric weights (clip_bary_pairs); masses in FP64.  Included
// by kernels.cuh.
//
// A CTA takes up to 32 tets through set-up, listing of the partial cells and
// clipping, phases of the whole CTA so that each one's code stays in the
// instruction cache.  A warp per tet, set up by one lane, had spent half its
// time on FP64 instructions of one or a few lanes and waited for instructions
// otherwise: a 256^3 clustered lattice 12.5 ms, now 2.6; a ragged patch call
// 107 us, now 34; the smallest boundary call 57 us, now 30.  What is left is
// latency: the set-up's chain of loads and FP64 operations, and lists of a few
// hundred cells shared by 8 warps.
#pragma once

namespace adeco {

// A tet being routed (shared memory): the FP32 vertex pairs hi + lo in the
// anchor frame, their planes and error band; FP64 planes for the cells the
// FP32 ones are unsure of, and the row bounds (made when a tet of the batch
// needs them; until then pn holds the vertices).
struct RouteTet {
    double pn[4][3], pd[4], pp[4], pm[4], rnx[4];
    double f6;
    const GridDesc *g;
    float4 plane[4];   // FP32 normal and offset
    float2 extent[4];  //   what the largest and the smallest corner of a cell add to the value at its origin
    float qf[4][3], ql[4][3], bmin[3], bmax[3], drcell[3], tol;
    int ex[3], lo[3];
};

constexpr int kRouteTets = 32;  // tets a CTA has set up at a time

struct RouteShared {
    RouteTet t[kRouteTets];
    // the tets with candidates, in order: the rows or cells of the tets up to
    // this one, and its slot
    int end[kRouteTets];
    uint8_t slot[kRouteTets];
    int total;   // rows and cells of all
    int cursor;  //   and the first not taken
    int rows;       // a tet is classified by rows
    int unsure[2];  // cells at the end of the list that the FP32 planes are unsure of (alternating as list.n)
    BaryList list;
    BaryPool pool[kWarps];
};

constexpr size_t kRouteSmem = sizeof(RouteShared);
static_assert(kRouteTets == 32, "a lane per tet, and 4 threads per tet, in the set-up");
static_assert(2 * (kRouteSmem + 1024) <= 228 * 1024, "two CTAs per SM");

// Tets with this many cells along x are classified by rows of cells (the
// bounds of 32 rows keep the FP64 pipe busy as long as 16 rounds of cells
// take), others cell by cell.  256^3 clustered lattice, all of the deposit,
// from 8 / 12 / 17 cells on: 36.0 / 36.1 / 35.6 ms.
constexpr int kRouteRow = 17;

// FP64 operations take their pipe 16 cycles each however many lanes take
// part: a tet's vertices and faces are made by 4 lanes, 8 tets a warp, and what
// is one per tet by a lane each.

// Vertex (and FP32 face) f = threadIdx.x & 3 of a tet, for candidate range [lo, hi].
__device__ __forceinline__ void route_setup(RouteTet &T, const float3 v[4], const int lo[3], const int hi[3],
                                            const GridDesc &g)
{
    const int f = threadIdx.x & 3;
    const float3 own = make_float3(sel4(f, v[0].x, v[1].x, v[2].x, v[3].x), sel4(f, v[0].y, v[1].y, v[2].y, v[3].y),
                                   sel4(f, v[0].z, v[1].z, v[2].z, v[3].z));
    float qf[3];
    float R = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double anchor = fma((double)lo[a], g.delta_d[a], g.gmin_d[a]);
        const double x = (a == 0) ? (double)own.x : ((a == 1) ? (double)own.y : (double)own.z);
        const double q = (x - anchor) * g.scale_d[a];
        T.pn[f][a] = q;
        qf[a] = __double2float_rn(q);
        T.qf[f][a] = qf[a];
        T.ql[f][a] = __double2float_rn(q - (double)qf[a]);
        R = fmaxf(fmaxf(R, (float)(hi[a] - lo[a] + 1)), fabsf(qf[a]));
    }
    R = fmaxf(R, __shfl_xor_sync(0xffffffffu, R, 1));
    R = fmaxf(R, __shfl_xor_sync(0xffffffffu, R, 2));
    // face f's vertices: 0 2 1, 0 3 2, 0 1 3, 1 2 3
    const int ia = f == 3, ib = f == 0 ? 2 : (f == 1 ? 3 : (f == 2 ? 1 : 2)), ic = f == 0 ? 1 : (f == 1 ? 2 : 3);
    float s1[3], s2[3], so[3], bmin[3], bmax[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        so[a] = __shfl_sync(0xffffffffu, qf[a], ia, 4);
        s1[a] = __shfl_sync(0xffffffffu, qf[a], ib, 4) - so[a];
        s2[a] = __shfl_sync(0xffffffffu, qf[a], ic, 4) - so[a];
        bmin[a] = fminf(qf[a], __shfl_xor_sync(0xffffffffu, qf[a], 1));
        bmin[a] = fminf(bmin[a], __shfl_xor_sync(0xffffffffu, bmin[a], 2));
        bmax[a] = fmaxf(qf[a], __shfl_xor_sync(0xffffffffu, qf[a], 1));
        bmax[a] = fmaxf(bmax[a], __shfl_xor_sync(0xffffffffu, bmax[a], 2));
    }
    const float nx = s1[1] * s2[2] - s1[2] * s2[1], ny = s1[2] * s2[0] - s1[0] * s2[2],
                nz = s1[0] * s2[1] - s1[1] * s2[0];
    const float pos = fmaxf(nx, 0.f) + fmaxf(ny, 0.f) + fmaxf(nz, 0.f);
    T.plane[f] = make_float4(nx, ny, nz, nx * so[0] + ny * so[1] + nz * so[2]);
    T.extent[f] = make_float2(pos, (nx + ny + nz) - pos);
    const float L1 = fmaxf(fmaxf(fabsf(s1[0]), fabsf(s1[1])), fabsf(s1[2]));
    const float L2 = fmaxf(fmaxf(fabsf(s2[0]), fabsf(s2[1])), fabsf(s2[2]));
    float tol = fmaxf(0.f, 1.0e-5f * L1 * L2 * (R + 1.f));
    tol = fmaxf(tol, __shfl_xor_sync(0xffffffffu, tol, 1));
    tol = fmaxf(tol, __shfl_xor_sync(0xffffffffu, tol, 2));
    if (f == 0) {
        T.g = &g;
        T.tol = tol;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (f == a) {
            T.ex[a] = hi[a] - lo[a] + 1;
            T.lo[a] = lo[a];
            T.bmin[a] = bmin[a];
            T.bmax[a] = bmax[a];
            T.drcell[a] = g.drcell[a];
        }
}

// FP64 planes of the tets set up, 4 lanes a tet (their vertices are in pn)
__device__ __forceinline__ void route_planes(RouteShared &S)
{
    if (threadIdx.x >= 4 * kRouteTets) return;  // whole warps
    RouteTet &T = S.t[threadIdx.x >> 2];
    const int f = threadIdx.x & 3;
    const int ia = f == 3, ib = f == 0 ? 2 : (f == 1 ? 3 : (f == 2 ? 1 : 2)), ic = f == 0 ? 1 : (f == 1 ? 2 : 3);
    double o[3], e1[3], e2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        o[a] = T.pn[ia][a];
        e1[a] = T.pn[ib][a] - o[a];
        e2[a] = T.pn[ic][a] - o[a];
    }
    __syncwarp();
    const double nx = e1[1] * e2[2] - e1[2] * e2[1], ny = e1[2] * e2[0] - e1[0] * e2[2],
                 nz = e1[0] * e2[1] - e1[1] * e2[0];
    T.pn[f][0] = nx;
    T.pn[f][1] = ny;
    T.pn[f][2] = nz;
    T.pd[f] = nx * o[0] + ny * o[1] + nz * o[2];
    T.pp[f] = fmax(nx, 0.0) + fmax(ny, 0.0) + fmax(nz, 0.0);
    T.pm[f] = fmin(nx, 0.0) + fmin(ny, 0.0) + fmin(nz, 0.0);
    const double nxr = nx * T.g->rcell[0];
    T.rnx[f] = nxr != 0.0 ? 1.0 / nxr : 0.0;
}

// Cell (a, b, k) of the routed tet: 0 outside, 1 holding the whole tet, 2
// inside the tet, 3 partial, 4 the FP32 planes are unsure (classify_pair's
// tests and error band).
__device__ __forceinline__ int route_classify(const RouteTet &T, int a, int b, int k)
{
    const float xa = (float)a, xb = (float)b, xk = (float)k;
    if (!(T.bmin[0] < xa + 1.f && xa < T.bmax[0] && T.bmin[1] < xb + 1.f && xb < T.bmax[1] && T.bmin[2] < xk + 1.f &&
          xk < T.bmax[2]))
        return 0;
    if (T.bmin[0] >= xa && T.bmax[0] <= xa + 1.f && T.bmin[1] >= xb && T.bmax[1] <= xb + 1.f && T.bmin[2] >= xk &&
        T.bmax[2] <= xk + 1.f)
        return 1;
    bool all_in = true, unsure = false;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const float4 n = T.plane[f];
        const float2 e = T.extent[f];
        const float base = fmaf(n.x, xa, fmaf(n.y, xb, fmaf(n.z, xk, -n.w)));
        const float mx = base + e.x, mn = base + e.y;
        if (mx < -T.tol) return 0;
        if (mx <= T.tol) unsure = true;
        if (mn > T.tol) continue;
        all_in = false;
        if (mn > -T.tol) unsure = true;
    }
    return unsure ? 4 : (all_in ? 2 : 3);
}

// The same from the FP64 planes
__device__ __forceinline__ int route_classify_fp64(const RouteTet &T, const GridDesc &g, int a, int b, int k)
{
    const double oa = a * g.rcell[0], ob = b * g.rcell[1], ok = k * g.rcell[2];
    bool all_in = true;
    for (int f = 0; f < 4; ++f) {
        const double base = T.pn[f][0] * oa + T.pn[f][1] * ob + T.pn[f][2] * ok - T.pd[f];
        if (base + T.pp[f] <= 0.0) return 0;
        if (!(base + T.pm[f] > 0.0)) all_in = false;
    }
    return all_in ? 2 : 3;
}

// Adds dm (in the grid's units) to cell (a, b, k) of the tet's range.
__device__ __forceinline__ void route_put(unsigned long long *out, const RouteTet &T, const GridDesc &g, int a, int b,
                                          int k, double dm)
{
    const unsigned long long fx = (unsigned long long)llrint(ldexp(dm, g.shift));
    if (fx)
        atomicAdd(out + g.out_offset + (T.lo[0] + a) +
                      (long long)g.dims * ((T.lo[1] + b) + (long long)g.dims * (T.lo[2] + k)),
                  fx);
}

// A row of cells (b, k) of a tet: the FP64 plane bounds, linear in the cell
// index and widened by a cell against rounding, skip the cells certainly
// outside and give the ones certainly inside, [li, hi]; the cells to classify
// are [a, a1) and [a2, a3].  False if the row has none of either.
__device__ __forceinline__ bool route_row(const RouteTet &T, const GridDesc &g, int b, int k, int &a, int &a1, int &a2,
                                          int &a3)
{
    const double ob = b * g.rcell[1], ok = k * g.rcell[2];
    double lo_c = 0.0, hi_c = T.ex[0] - 1, lo_i = 0.0, hi_i = T.ex[0] - 1;
    bool none = false, no_in = false;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const double nx = T.pn[f][0];
        const double K = T.pn[f][1] * ob + T.pn[f][2] * ok - T.pd[f];
        if (nx > 0.0) {
            lo_c = fmax(lo_c, floor(-(K + T.pp[f]) * T.rnx[f]) - 1.0);
            lo_i = fmax(lo_i, floor(-(K + T.pm[f]) * T.rnx[f]) + 2.0);
        } else if (nx < 0.0) {
            hi_c = fmin(hi_c, ceil(-(K + T.pp[f]) * T.rnx[f]) + 1.0);
            hi_i = fmin(hi_i, ceil(-(K + T.pm[f]) * T.rnx[f]) - 2.0);
        } else {
            none = none || !(K + T.pp[f] > 0.0);
            no_in = no_in || !(K + T.pm[f] > 0.0);
        }
    }
    if (none) return false;
    const int lc = (int)fmax(lo_c, 0.0), hc = (int)fmin(hi_c, (double)(T.ex[0] - 1));
    int li = (int)fmax(lo_i, (double)lc), hi = (int)fmin(hi_i, (double)hc);
    if (no_in || li > hi) {
        li = hc + 1;
        hi = hc;
    }
    a = lc;
    a1 = li;
    a2 = hi + 1;
    a3 = hc;
    return true;
}

// Set up tets first, first + step, ... (n of them) of the list (the whole CTA).
__device__ __forceinline__ void route_setup_tets(const DepositParams &P, RouteShared &S, unsigned long long first,
                                                 unsigned long long step, int n)
{
    const int slot = threadIdx.x >> 2;
    if (threadIdx.x < 4 * kRouteTets) {  // whole warps
        const bool has = slot < n;
        const unsigned long long entry = P.route[first + step * (has ? slot : 0)];
        const Item it = P.items[entry >> 16];
        const int local = (int)(entry & 0xffff), c = local / 6, t = local % 6;
        const int vx = it.nv & 0xff, vy = (it.nv >> 8) & 0xff;
        const int cvx = vx - 1, cvy = vy - 1;
        const int ci = c % cvx, r = c / cvx, cj = r % cvy, ck = r / cvy;
        float3 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int3 o = corner_offset(P.order, tet_conn(t, q));
            const long long gi = it.base + (ci + o.x) + P.stride_y * (cj + o.y) + P.stride_z * (ck + o.z);
            if (P.src_kind == SRC_LATTICE_F4) {
                const float4 p = __ldg(reinterpret_cast<const float4 *>(P.src) + gi);
                v[q] = make_float3(p.x, p.y, p.z);
            } else {
                const float *s = reinterpret_cast<const float *>(P.src) + 3 * gi;
                v[q] = make_float3(__ldg(s), __ldg(s + 1), __ldg(s + 2));
            }
        }
        if (vol6_sign_ref(vol6_exact(v[0], v[1], v[2], v[3])) < 0) {
            const float3 tmp = v[0];
            v[0] = v[3];
            v[3] = tmp;
        }
        const GridDesc &g = P.grids[it.grid];
        int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
        const bool some = candidate_range(v, g, lo, hi) && tile_clamp(g, lo, hi) && has;
        __syncwarp();
        route_setup(S.t[slot], v, lo, hi, g);
        if ((threadIdx.x & 3) == 0) {
            // (at most 2^25 cells a tet, so 2^30 of all)
            const int ex = hi[0] - lo[0] + 1, rows = (hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1);
            S.end[slot] = some ? (ex >= kRouteRow ? rows : ex * rows) : 0;
        }
    }
    if (threadIdx.x == 0) S.cursor = 0;
    __syncthreads();
    if (threadIdx.x < 32) {  // a lane per tet
        const int k = threadIdx.x;
        RouteTet &T = S.t[k];
        T.f6 = T.g->mass_factor / fabs(vol6_fast<double>(T.pn[0], T.pn[1], T.pn[2], T.pn[3]));
        const int own = S.end[k];
        const unsigned some = __ballot_sync(0xffffffffu, own > 0);
        const bool rows = __any_sync(0xffffffffu, own && T.ex[0] >= kRouteRow);
        int u = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, u, o);
            if (k >= o) u += y;
        }
        S.end[k] = INT_MAX;
        __syncwarp();
        if (own) {
            const int m = __popc(some & ((1u << k) - 1));
            S.end[m] = u;
            S.slot[m] = (uint8_t)k;
        }
        if (k == 31) {
            S.total = u;
            S.rows = rows;
        }
    }
    __syncthreads();
}

// bitwise or over the warp (the host checks' compiler target has no reduction instruction)
__device__ __forceinline__ unsigned warp_or(unsigned v)
{
#if !defined(__CUDA_ARCH__) || __CUDA_ARCH__ >= 800
    return __reduce_or_sync(0xffffffffu, v);
#else
    for (int o = 16; o > 0; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
    return v;
#endif
}

// A lane's cells in hand: [a, a1) and [a2, a3] of row (b, k) of tet s, cell a
// of which is number base + a of the tet's box.
struct RouteRow {
    int s, b, k, base, a, a1, a2, a3;
};

// Lists the partial cells of the tets set up, and at the list's end the cells
// the FP32 planes are unsure of: their FP64 test, for a few lanes of nearly
// every round here, kept the FP64 pipe busy for most of the phase.  The rows
// and cells of all tets are numbered through and taken 32 at a time, a lane
// each, until none is left or the list might not hold another round of every
// warp; a round classifies a cell of each lane.  Cells holding the tet or inside
// it are deposited at once.  Cells in hand carry over to the next call; true
// while this warp has any.
__device__ __forceinline__ bool route_list(const DepositParams &P, RouteShared &S, int *list_n, int *unsure_n, bool busy,
                                           RouteRow &w, unsigned &n_cand, unsigned &n_part, unsigned &n64)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1;
    const int end = S.end[lane], total = S.total;
    for (;;) {
        int c0 = 0;
        if (lane == 0)
            c0 = *(volatile int *)list_n + *(volatile int *)unsure_n > kBaryPairs - kThreads
                     ? -1
                     : (busy ? 0 : atomicAdd(&S.cursor, 32));
        c0 = __shfl_sync(0xffffffffu, c0, 0);
        if (c0 < 0 || c0 >= total) return busy;
        if (!busy) {
            // the lane's tet: the first one's, and one more for each that ends before the lane's number
            const int first = __popc(__ballot_sync(0xffffffffu, end <= c0));
            const unsigned ends = warp_or(end > c0 && end - c0 < 32 ? 1u << (end - c0) : 0u);
            const int m = first + __popc(ends & (lt << 1 | 1));
            const int before = __shfl_sync(0xffffffffu, end, (m - 1) & 31);
            const int e = c0 + lane - (m ? before : 0);
            w.a = w.a1 = w.a2 = 0;
            w.a3 = -1;
            if (c0 + lane < total) {
                w.s = S.slot[m];
                const RouteTet &T = S.t[w.s];
                if (T.ex[0] >= kRouteRow) {
                    const int3 c = box_cell(T.ex[1], T.ex[2], e);
                    w.b = c.x;
                    w.k = c.y;
                    w.base = T.ex[0] * e;
                    const GridDesc &g = *T.g;
                    if (route_row(T, g, w.b, w.k, w.a, w.a1, w.a2, w.a3)) {
                        const double inside6 = 6.0 * T.f6;
                        for (int x = w.a1; x < w.a2; ++x) route_put(P.out, T, g, x, w.b, w.k, inside6);
                        n_cand += max(w.a2 - w.a1, 0);
                    }
                } else {
                    const int3 c = box_cell(T.ex[0], T.ex[1], e);
                    w.a = c.x;
                    w.a1 = c.x + 1;
                    w.b = c.y;
                    w.k = c.z;
                    w.base = e - c.x;
                }
            }
        }
        int cls = 0, a = 0;
        if (w.a < w.a1 || w.a2 <= w.a3) {
            a = w.a < w.a1 ? w.a++ : w.a2++;
            const RouteTet &T = S.t[w.s];
            ++n_cand;
            cls = route_classify(T, a, w.b, w.k);
            if (cls == 1 || cls == 2)
                route_put(P.out, T, *T.g, a, w.b, w.k, cls == 1 ? (double)T.g->tet_mass : 6.0 * T.f6);
        }
        const unsigned part = __ballot_sync(0xffffffffu, cls == 3), unsure = __ballot_sync(0xffffffffu, cls == 4);
        int at = 0;
        if (lane == 0 && part) at = atomicAdd(list_n, __popc(part));
        if (lane == 1 && unsure) at = atomicAdd(unsure_n, __popc(unsure));
        const int end_at = kBaryPairs - 1 - (__shfl_sync(0xffffffffu, at, 1) + __popc(unsure & lt));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(part & lt);
        if (cls >= 3) {
            if (cls == 4) at = end_at;
            S.list.cell[at] = (uint32_t)(w.base + a);
            S.list.tet[at] = (uint8_t)w.s;
            ++(cls == 3 ? n_part : n64);
        }
        busy = __any_sync(0xffffffffu, w.a < w.a1 || w.a2 <= w.a3);
    }
}

// The nu unsure cells at the list's end, a thread each, by the FP64 planes: the
// partial ones are listed, those inside deposited.  256 at a time from the
// lowest: what is listed then takes places that are read already, since a
// partial cell comes for each unsure one at most.
__device__ __forceinline__ void route_resolve(const DepositParams &P, RouteShared &S, int *list_n, int nu,
                                              unsigned &n_part)
{
    const unsigned lt = (1u << (threadIdx.x & 31)) - 1;
    for (int i = 0; i < nu; i += kThreads) {
        const int j = i + (int)threadIdx.x;
        int cls = 0, s = 0;
        uint32_t cell = 0;
        if (j < nu) {
            cell = S.list.cell[kBaryPairs - nu + j];
            s = S.list.tet[kBaryPairs - nu + j];
            const RouteTet &T = S.t[s];
            const GridDesc &g = *T.g;
            const int3 c = box_cell(T.ex[0], T.ex[1], (int)cell);
            cls = route_classify_fp64(T, g, c.x, c.y, c.z);
            if (cls == 2) route_put(P.out, T, g, c.x, c.y, c.z, 6.0 * T.f6);
        }
        __syncthreads();
        const unsigned part = __ballot_sync(0xffffffffu, cls == 3);
        int at = 0;
        if ((threadIdx.x & 31) == 0 && part) at = atomicAdd(list_n, __popc(part));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(part & lt);
        if (cls == 3) {
            S.list.cell[at] = cell;
            S.list.tet[at] = (uint8_t)s;
            ++n_part;
        }
    }
}

// The tets deposit_mixed_kernel listed, up to kRouteTets of a CTA at a time:
// set-up, listing of the partial cells and clipping are phases of the whole
// CTA.
__global__ void __launch_bounds__(kThreads, 2) route_fp64_kernel(DepositParams P)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RouteShared &S = *reinterpret_cast<RouteShared *>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long count = *P.route_count;
    const unsigned long long n = count < P.route_cap ? count : P.route_cap;
    // batches of at most kRouteTets, fewer when there are fewer tets than that
    // for every CTA; a batch's tets are spread over the list, since neighbours
    // in the list are of similar size
    const unsigned long long share = (n + gridDim.x - 1) / gridDim.x;
    const unsigned per = share < kRouteTets ? max((unsigned)share, 1u) : kRouteTets;
    const unsigned long long batches = (n + per - 1) / per;
    unsigned cand = 0, part = 0, n64 = 0;
    int turn = 0;  // the pair list's counters in use
    if (threadIdx.x == 0) S.list.n[0] = S.list.next[0] = S.unsure[0] = 0;
    for (unsigned long long batch = blockIdx.x; batch < batches; batch += gridDim.x) {
        const int nt = (int)((n - batch + batches - 1) / batches);
        route_setup_tets(P, S, batch, batches, nt);
        bool planes = S.rows != 0;
        if (planes) {
            route_planes(S);
            __syncthreads();
        }
        RouteRow w = {0, 0, 0, 0, 0, 0, 0, -1};
        bool busy = false, left = true;
        while (left) {
            busy = route_list(P, S, &S.list.n[turn], &S.unsure[turn], busy, w, cand, part, n64);
            left = __syncthreads_or(busy) || S.cursor < S.total;
            const int nu = S.unsure[turn];
            if (threadIdx.x == 0) S.list.n[turn ^ 1] = S.list.next[turn ^ 1] = S.unsure[turn ^ 1] = 0;  // the next list's
            if (nu) {
                if (!planes) {
                    route_planes(S);
                    __syncthreads();
                    planes = true;
                }
                route_resolve(P, S, &S.list.n[turn], nu, part);
                __syncthreads();
            }
            const int np = S.list.n[turn];
            uint64_t mine = clip_bary_pairs(
                S.pool[warp], S.list, &S.list.next[turn], np,
                [&](int j, float *x) {
                    const RouteTet &T = S.t[S.list.tet[j]];
                    const int3 c = box_cell(T.ex[0], T.ex[1], (int)S.list.cell[j]);
                    // coordinates in the cell's mirrored frame along axes whose
                    // lower face the tet does not reach (as piece_coords); the
                    // shares come from the weights, so no reordering is needed
                    const int cc[3] = {c.x, c.y, c.z};
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        const bool flip = T.bmin[i] > (float)cc[i];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            x[3 * q + i] = cell_coord_sel(T.qf[q][i], T.ql[q][i], cc[i], T.drcell[i], flip);
                    }
                });
            // the masses of this warp's pairs: share of the tet times its exact mass
            while (mine) {
                const int j = 32 * (__ffsll((long long)mine) - 1) + lane;
                mine &= mine - 1;
                if (j < np) {
                    const RouteTet &T = S.t[S.list.tet[j]];
                    const GridDesc &g = *T.g;
                    const int3 c = box_cell(T.ex[0], T.ex[1], (int)S.list.cell[j]);
                    const double dm = ldexp((double)S.list.volume(j), -kVolShift) * g.mass_factor;
                    if (dm > 0.0) route_put(P.out, T, g, c.x, c.y, c.z, dm);
                }
            }
            turn ^= 1;
            __syncthreads();
        }
    }
    if (P.stats) {
        warp_stat(P.stats, ST_CAND, cand);
        warp_stat(P.stats, ST_PARTIAL, part);
        warp_stat(P.stats, ST_FP64, n64);
    }
}

}  // namespace adeco

// Lattice form of the fused step, for meshes that are uniform grids.
//
// A uniform NE/NS mesh (one cell size, one side length per orientation,
// one side per face) is a 2-D lattice whatever its numbering. The planner
// below recognises it from the mesh tables and numbers it into a padded
// lattice: a border of holes (2 columns west, 2 rows south) and padding up
// to whole strips of 28 columns and chunks of rows (3 rows above the last
// chunk). During a batch the library keeps its own lattice-ordered copies
// of the state (depth and side discharges double-buffered, rain time,
// infiltration, extrema), gathered from the caller's arrays at the batch
// start and scattered back at its end. Inside the batch every neighbour is
// found by arithmetic: no index tables, rows of 32 cells per warp,
// coalesced loads.
//
// One step is two launches. k_lattice_march: each warp marches up a strip
// of the lattice with the rows it needs in registers and does, row by row,
// what the reference's passes do (solver_compact.py:439-641): momentum q*,
// donor factors, final discharges, sources and depth update, extrema,
// budget terms and the CFL candidates of the sides inside its strip and
// chunk; it writes its counters, its CFL minimum and its edge columns to
// per-warp records. k_lattice_close: those records, the CFL candidates of
// the sides on strip and chunk edges, the canonical 256-cell budget trees
// of the blocks the step touched, and in its last block the commit of the
// step and the prepare of the next. Each quantity is computed in the
// reference's operation order with the same expressions as the tiled and
// multi-pass steps, so the three forms and the CPU restatement agree bit
// for bit.
//
// Budget terms are sums over the reference's 256-cell blocks of global ids
// (ei // 256), which a lattice strip does not follow: the march writes each
// nonzero per-cell term into a scratch array by global id and marks its
// block; the close pass reduces the marked blocks with the canonical tree
// and clears them.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "nhf_common.cuh"
#include "nhf_math.cuh"

namespace nhf {
namespace {

constexpr int kLanes = 32;                        // a warp marches a strip of 32 lattice columns
constexpr int kOut = 28;                          // and owns the 28 of lanes 2..29
constexpr int kWarps = 8, kNT = kLanes * kWarps;  // a block: up to 8 strips side by side
constexpr int kWest = 2;                          // border columns west of cell column 0

// A value of a lattice array at a byte offset: lattice indices are under 2^30, so
// 32-bit offsets reach every point and a load needs no 64-bit arithmetic.
template <typename T>
__device__ __forceinline__ T at(const T *base, uint32_t bytes)
{
    return __ldg(reinterpret_cast<const T *>(reinterpret_cast<const char *>(base) + bytes));
}
template <typename T>  // of an array the march writes
__device__ __forceinline__ T get(const T *base, uint32_t bytes)
{
    return *reinterpret_cast<const T *>(reinterpret_cast<const char *>(base) + bytes);
}
template <typename T>
__device__ __forceinline__ void put(T *base, uint32_t bytes, T v)
{
    *reinterpret_cast<T *>(reinterpret_cast<char *>(base) + bytes) = v;
}

// x / b for a fixed b: the product with 1 / b where that is exact (b a power of
// two; inverse 0 elsewhere).
__device__ __forceinline__ real over(real x, real b, real inverse) { return inverse != RC(0) ? x * inverse : x / b; }

// Momentum (solver_compact.py:439-486) of one side from the cells either
// side of it (a: lower, b: higher) and the side's discharge xq and Manning
// n; the same expressions as the tiled step's P1. kPlain: both cells are live.
template <bool kPlain>
__device__ __forceinline__ real lattice_momentum(const Dev &d, real dt, real za, real ha, real zb, real hb,
                                                 bool live_a, bool live_b, real xq, real n,
                                                 const int32_t *side_ids, uint32_t off, real sdc, real inverse)
{
    const real hl = za + ha, hr = zb + hb;
    const real xwh = rmax(hl, hr) - rmaxc(rmax(za, zb), kDh);
    real new_q = RC(0);
    if (!(xwh < d.min_h)) {
        const bool exterior = !kPlain && live_a != live_b;
        const real slope = d.neg_g * (hr - hl);
        const real xdq = (exterior ? slope / d.sdc[at(side_ids, off)] : over(slope, sdc, inverse)) *
                         rmaxc(xwh, RC(0)) * dt;
        real ratio = RC(0);
        if (xq != RC(0)) ratio = xq / friction_pow_real(rmaxc(xwh, RC(0.00001)));
        const real xf = RC(1) + d.g * dt * (n * n) * fabs(ratio);
        const real nb = RC(0) + RC(0);
        new_q = (d.sita * xq + d.half_rest * nb + xdq) / xf;
        if (!kPlain) new_q *= exterior ? RC(0) : RC(1);
    }
    return new_q;
}

// Donor factor (solver_compact.py:491-514) of the cell at offset `off`
// (boundary id bi, rain rate rainq) from its depth and the q* of its west,
// east, south and north faces; sets ``limited`` when the outflow had to be
// scaled. kPlain: no boundary cell.
template <bool kPlain>
__device__ __forceinline__ real lattice_donor(const Dev &d, const LatticePlan &P, uint32_t off, int bi, real h, real dt,
                                              real rainq, real qw, real qe, real qs, real qn, bool &limited)
{
    const nhf_mesh &m = d.m;
    int kind = -1;
    real discharge = RC(0);
    if (!kPlain && bi >= 0) {
        kind = m.kind[bi];
        if (kind == 1) discharge = d.values[bi] * m.weight[at(P.cell, off)];
    }
    const real positive = kPlain ? RC(0) : (RC(0) + rmaxc(discharge, RC(0))) * dt;
    const real area = P.area;
    const real available = h * area + positive + rainq * dt * area;
    real outgoing = kPlain ? RC(0) : (RC(0) + rmaxc(-discharge, RC(0))) * dt;
    outgoing += rmaxc(-(qw * P.len_v), RC(0)) * dt;
    outgoing += rmaxc(qe * P.len_v, RC(0)) * dt;
    outgoing += rmaxc(-(qs * P.len_h), RC(0)) * dt;
    outgoing += rmaxc(qn * P.len_h, RC(0)) * dt;
    real sc = RC(1);
    limited = false;
    if (outgoing > available && kind != 0) {
        sc = available / outgoing;
        limited = true;
    }
    return sc;
}

// The per-cell inputs of a depth update, loaded a row ahead of their use.
struct LatticeCell {
    int g, bi;
    real rain_time, infil, max_speed, max_depth, f0, fc, k;
};

// A nonzero budget term of cell g into the scratch; the cell's block is marked
// (term 0, which every infiltrating cell has, by a plain byte store).
__device__ __forceinline__ void lattice_term(const LatticePlan &P, size_t e, int t, int g, real v)
{
    P.terms[t * e + g] = v;
    if (t == 0) P.touched_rain[g >> 8] = 1;
    else atomicOr(&P.touched[g >> 8], 1u << t);
}

// Sources and depth update (solver_compact.py:525-610) of the cell at offset
// `off` from its old depth, its donor factor and the final discharges of its
// four faces; writes the cell's rain time, infiltration, extrema and budget
// terms and returns the new depth.
template <bool kPlain>
__device__ __forceinline__ real lattice_update(const Dev &d, const LatticePlan &P, uint32_t off, real dt, real rainq,
                                               real previous, real z, real sc, real fw, real fe, real fs, real fn,
                                               const LatticeCell &k, const uint32_t *step_end)
{
    const nhf_mesh &m = d.m;
    const int bi = kPlain ? -1 : k.bi;
    const int B = m.b_num;
    const int kind = bi >= 0 ? m.kind[bi] : -1;
    const real pq = RC(0);
    const real pipe = rmax(pq, RC(0)) + rmin(pq, RC(0)) * sc;
    real discharge = RC(0), t_discharge = RC(0);
    if (!kPlain && kind == 1) {
        real requested = d.values[bi] * m.weight[at(P.cell, off)];
        discharge = rmaxc(requested, RC(0)) + rmin(requested, RC(0)) * sc;
        t_discharge = discharge * dt;
    }
    const real ssq = pipe + discharge;
    real infil = k.infil;
    if (rainq > RC(0)) {
        const real rt = k.rain_time + dt;
        put(P.rain_time, off, rt);
        // without Horton classes every f0, fc and k is zero (checked by the planner)
        const real diff = k.f0 - k.fc;
        infil = diff == RC(0) ? k.fc + RC(0) : k.fc + diff * exp_real(-k.k * rt / RC(3600.0));
        if (__float_as_uint(infil) != __float_as_uint(k.infil)) put(P.infil, off, infil);
    }
    const real ql = RC(0) + fw * P.len_v, qr = RC(0) + fe * P.len_v;
    const real qb = RC(0) + fs * P.len_h, qt = RC(0) + fn * P.len_h;
    const real tq = ql - qr + qb - qt + ssq;
    const real ea = P.area;
    const real rain_depth = rainq * dt;
    const real flux = tq * dt;
    const real increment = (flux == RC(0) ? flux : over(flux, ea, P.inv_area)) + rain_depth;
    real raw_depth = previous + increment;
    const real removed = rmin(infil * dt, rmaxc(raw_depth, RC(0)));
    raw_depth -= removed;
    const real floor_v = rmaxc(-raw_depth, RC(0));
    const real depth = kind == 0 ? rmaxc(d.level_values[bi] - z, RC(0)) : rmaxc(raw_depth, RC(0));
    const real fastest = fastest_speed(depth >= d.min_h, ql + qr, qb + qt, P.height, P.width, rmaxc(depth, RC(0.01)),
                                       k.max_speed);
    if (fastest > k.max_speed) put(P.max_speed, off, fastest);
    if (depth > k.max_depth) {
        put(P.max_depth, off, depth);
        put(P.peak_hi, off, __ldg(step_end));  // the clock words are not written during the march
        put(P.peak_lo, off, __ldg(step_end + 1));
    }
    // budget terms of this cell by global id: 0 removed, 1 / 2 bed clamp
    // off / on level cells, 3 pipe (none), 4 + 5 b + k level, 4 + 5 B + b discharge
    const size_t e = (size_t)m.e_num;
    const real removed_v = removed * ea, floor_a = floor_v * ea;
    if (removed_v != RC(0)) lattice_term(P, e, 0, P.horton ? k.g : at(P.cell, off), removed_v);
    if (floor_a != RC(0)) lattice_term(P, e, kind == 0 ? 2 : 1, at(P.cell, off), floor_a);
    if (!kPlain && kind == 0) {
        const real level[5] = {(depth - previous) * ea, -(ql - qr + qb - qt) * dt, -pipe * dt, -rain_depth * ea,
                               removed * ea};
        for (int q5 = 0; q5 < 5; ++q5)
            if (level[q5] != RC(0)) lattice_term(P, e, 4 + 5 * bi + q5, at(P.cell, off), level[q5]);
    }
    if (!kPlain && kind == 1 && t_discharge != RC(0)) lattice_term(P, e, 4 + 5 * B + bi, at(P.cell, off), t_discharge);
    return depth;
}

// CFL candidate (solver_compact.py:617-641) of one interior side, folded
// into the running minimum key (dt bits << 32 | side id). A side at the face
// depth's floor with no discharge is left to the dry key, the least key of an
// all-dry state, which the close pass folds in: no side's value is above its
// dry one, so where the minimum is that small the dry key's sides all attain
// it. Only a candidate that may be at or below the minimum is formed exactly,
// and only then is the side id read.
__device__ __forceinline__ void lattice_cfl(const Dev &d, real len, real q, real za, real ha, real zb, real hb,
                                            const int32_t *side_ids, uint32_t off, unsigned long long &best)
{
    const real head = rmax(za + ha, zb + hb);
    const real fd = rmaxc(head - rmaxc(rmax(za, zb), kDh), RC(0.01));
    if (fd == RC(0.01) && q == RC(0)) return;
    if (cfl_above(d.afa * len, d.g, q, fd, __uint_as_float((uint32_t)(best >> 32)))) return;
    const uint32_t bits = __float_as_uint(cfl_value(d.afa, d.g, len, q, fd));
    if (bits <= (uint32_t)(best >> 32)) {
        const unsigned long long key = ((unsigned long long)bits << 32) | (unsigned)at(side_ids, off);
        best = key < best ? key : best;
    }
}

// The state of buffer `p`, for rescan_cfl.
struct LatticeState {
    const LatticePlan *P;
    int p;
    __device__ __forceinline__ real depth(int cell) const { return __ldcg(P->h[p] + P->glat[cell]); }
    __device__ __forceinline__ real q(int side) const
    {
        const int at = P->gside[side];
        return __ldcg(((at & 1) ? P->qh[p] : P->qv[p]) + (at >> 1));
    }
};

// prepare_step (solver_compact.py:364-382) with the state in lattice order.
__device__ __noinline__ void lattice_prepare(const Dev &d, Ctl *c)
{
    const nhf_mesh &m = d.m;
    const LatticePlan &P = d.lat;
    clock_choose(d.min_dt, c, (float)c->ndt, c->trace + c->slot * NHF_TRACE_COLS);
    if (!c->active) return;
    c->limited_cells = 0; c->limited_faces = 0;
    c->min_scale_bits = real_bits(RC(1.0));
    c->wet = 0;
    for (int bi = 0; bi < m.b_num; ++bi) {
        d.values[bi] = d.coef[2 * bi] + d.coef[2 * bi + 1] * ((real)c->local + (real)c->dt / RC(2.0));
        d.level_values[bi] = d.coef[2 * bi] + d.coef[2 * bi + 1] * (real)c->end_local;
    }
    if (c->ndt < c->limit_value[0]) {
        const int si = c->cfl_arg;
        const int el = m.topology[3 * si + 1], eh = m.topology[3 * si + 2];
        const real *h = P.h[c->parity];
        const real de = el ? __ldcg(h + P.glat[el]) : m.depth[0];
        const real dh = eh ? __ldcg(h + P.glat[eh]) : m.depth[0];
        real fd = RC(0), q = m.q[0];
        if (si) {
            fd = cfl_face_depth(m.bed[el], de, m.bed[eh], dh);
            const int gs = P.gside[si];
            q = __ldcg(((gs & 1) ? P.qh[c->parity] : P.qv[c->parity]) + (gs >> 1));
        }
        c->limit_value[0] = c->ndt;
        c->limit_value[1] = de; c->limit_value[2] = dh;
        c->limit_value[3] = fd;
        c->limit_value[4] = q / rmax(fd, RC(1e-30));
        c->limit_ids[0] = si; c->limit_ids[1] = el; c->limit_ids[2] = eh;
    }
}
// The rows of one warp's strip and chunk (k_lattice_march). kPlain: every cell
// the warp looks at is live and off the boundaries, which holds for all but
// the strips and chunks at the domain's edge, so liveness, boundary ids and
// exterior sides drop out.
template <int kParity, bool kPlain>
__device__ __forceinline__ void lattice_rows(const Dev &d, const int strip, const int chunk, uint32_t &counts,
                                             uint32_t &min_bits, unsigned long long &best)
{
    constexpr unsigned kAll = 0xffffffffu;
    const LatticePlan &P = d.lat;
    const Ctl *c = d.ctl;
    const real dt = c->dt;
    const bool raining = c->raining != 0;
    const bool horton = raining && P.horton, keep_idle = *P.odd == 0 && d.min_h > RC(0);
    const real one_rate = raining && !P.rain_cells ? d.rain_rates[0] : RC(0);
    const real *h_in = P.h[kParity], *qv_in = P.qv[kParity], *qh_in = P.qh[kParity];
    real *h_out = P.h[1 - kParity], *qv_out = P.qv[1 - kParity], *qh_out = P.qh[1 - kParity];
    const int lane = threadIdx.x & 31;
    const bool own = lane >= 2 && lane < 2 + kOut;
    const int y0 = 2 + chunk * P.rows, y1 = y0 + P.rows;  // the rows this warp updates
    const uint32_t row = 4u * (uint32_t)P.lx;
    auto rate_at = [&](uint32_t off) { return raining && P.rain_cells ? at(P.rate, off) : one_rate; };
    auto live_at = [&](uint32_t off) { return kPlain || at(P.live, off >> 2) != 0; };
    auto bi_at = [&](uint32_t off) { return kPlain ? -1 : (int)at(P.bi, off >> 1); };
    // iteration y holds row y (h0 z0 l0), row y + 1 (h1 z1 l1), row y + 2
    // (h2 z2 l2), the inputs of the south side of row y + 2 (xs ns), of
    // the west side of row y + 1 (xw nw), the boundary id and rain rate of
    // row y + 1 (b1 r1), the rate of row y (r0) and the update inputs of row
    // y (k0, unless the whole warp's row is idle); it loads row y + 3 and
    // the side inputs first, the update inputs of row y + 1 last
    uint32_t o1 = 4u * ((uint32_t)(y0 - 2) * (uint32_t)P.lx + (uint32_t)(strip * kOut + lane));
    uint32_t o2 = o1 + row;
    real h1 = at(h_in, o1), z1 = at(P.z, o1), h2 = at(h_in, o2), z2 = at(P.z, o2);
    bool l1 = live_at(o1), l2 = live_at(o2);
    real xs = at(qh_in, o2), ns = at(P.nh, o2), xw = at(qv_in, o1), nw = at(P.nv, o1);
    int b1 = bi_at(o1);
    real r1 = rate_at(o1), r0 = RC(0);
    LatticeCell k0{0, -1, RC(0), RC(0), RC(0), RC(0), RC(0), RC(0), RC(0)};
    bool busy = false;
    real h0 = RC(0), z0 = RC(0), hm = RC(0), zm = RC(0);
    bool l0 = kPlain, lm = kPlain;
    real qs1 = RC(0), qw0 = RC(0), d0 = RC(0), fs0 = RC(0);  // q* south y+1, q* west y, donor y, final south y
    for (int y = y0 - 3; y < y1; ++y) {
        const uint32_t o0 = o1 - row, o3 = o2 + row;
        // what iteration y + 1 needs
        const real h3 = at(h_in, o3), z3 = at(P.z, o3);
        const bool l3 = live_at(o3);
        const real xs3 = at(qh_in, o3), ns3 = at(P.nh, o3);
        const real xw2 = at(qv_in, o2), nw2 = at(P.nv, o2);
        const int b2 = bi_at(o2);
        const real r2 = rate_at(o2);
        // q* of the south side of row y + 2 and of the west side of row y + 1
        real qs2 = RC(0);
        if (kPlain || l1 || l2)
            qs2 = lattice_momentum<kPlain>(d, dt, z1, h1, z2, h2, l1, l2, xs, ns, P.side_h, o2, P.sdc_h, P.inv_sdc_h);
        const real hw = __shfl_up_sync(kAll, h1, 1), zw = __shfl_up_sync(kAll, z1, 1);
        const bool lw = kPlain || __shfl_up_sync(kAll, (int)l1, 1) != 0;
        real qw1 = RC(0);
        if (lane > 0 && (kPlain || lw || l1))
            qw1 = lattice_momentum<kPlain>(d, dt, zw, hw, z1, h1, lw, l1, xw, nw, P.side_v, o1, P.sdc_v, P.inv_sdc_v);
        const real qe1 = __shfl_down_sync(kAll, qw1, 1);
        const bool out1 = own && y + 1 >= y0 && y + 1 < y1, out0 = own && y >= y0;
        // donor factor of row y + 1 (holes: the sentinel's factor 0)
        real d1 = RC(0);
        if (kPlain || l1) {
            bool limited;
            d1 = lattice_donor<kPlain>(d, P, o1, b1, h1, dt, r1, qw1, qe1, qs1, qs2, limited);
            if (limited && out1) {
                counts += 1u;
                const uint32_t bits = __float_as_uint(d1);
                min_bits = bits < min_bits ? bits : min_bits;
            }
        }
        // final discharge of the south side of row y + 1 and the west side of row y
        const real ss = qs1 >= RC(0) ? d0 : d1;
        const real fs1 = qs1 * ss;
        if (out1 && qs1 != RC(0) && ss < RC(1)) counts += 1u << 10;
        const real dwest = __shfl_up_sync(kAll, d0, 1);
        const real sw = qw0 >= RC(0) ? dwest : d0;
        const real fw0 = qw0 * sw;
        if (out0 && qw0 != RC(0) && sw < RC(1)) counts += 1u << 10;
        const real fe0 = __shfl_down_sync(kAll, fw0, 1);
        // update of row y; an idle row stays dry
        real hn = h0;
        if (out0 && (kPlain || l0)) {
            hn = RC(0);
            if (!kPlain || busy) {
                hn = lattice_update<kPlain>(d, P, o0, dt, r0, h0, z0, d0, fw0, fe0, fs0, fs1, k0, c->step_end);
                if (hn >= d.min_h) counts += 1u << 20;
            }
            put(h_out, o0, hn);
        }
        const real hnw = __shfl_up_sync(kAll, hn, 1), zw0 = __shfl_up_sync(kAll, z0, 1);
        const bool lw0 = kPlain || __shfl_up_sync(kAll, (int)l0, 1) != 0;
        if (out0) {
            if (kPlain || l0 || lw0) put(qv_out, o0, fw0);
            if (kPlain || l0 || lm) put(qh_out, o0, fs0);
            // the strip's edge cells for the close pass: the first column
            // (new depth, bed, discharge of its west side, liveness) and
            // the last (new depth, -1 for a hole, and bed)
            const size_t e_at = (size_t)strip * P.chunks * P.rows + (y - 2);
            if (lane == 2) P.edge_first[e_at] = make_float4(hn, z0, fw0, kPlain || l0 ? 1.0f : 0.0f);
            if (lane == 1 + kOut) P.edge_last[e_at] = make_float2(kPlain || l0 ? hn : -1.0f, z0);
            // interior sides both of whose cells this warp updated
            if ((kPlain || (l0 && lw0)) && lane > 2) lattice_cfl(d, P.len_v, fw0, zw0, hnw, z0, hn, P.side_v, o0, best);
            if ((kPlain || (l0 && lm)) && y > y0) lattice_cfl(d, P.len_h, fs0, zm, hm, z0, hn, P.side_h, o0, best);
        }
        // the update inputs of row y + 1, half an iteration ahead of their
        // use; none for a row whose cells are dry and stay dry (no rain, no
        // discharge on any side), which saves their 20 bytes a cell
        k0 = LatticeCell{0, b1, RC(0), RC(0), RC(0), RC(0), RC(0), RC(0), RC(0)};
        const bool moves = qw1 != RC(0) || qe1 != RC(0) || qs1 != RC(0) || qs2 != RC(0) || h1 != RC(0) || r1 != RC(0);
        busy = __any_sync(kAll, own && moves) || !keep_idle;
        if (own && (kPlain ? busy : l1) && y + 1 >= y0 && y + 1 < y1) {
            k0.infil = get(P.infil, o1);
            k0.max_speed = get(P.max_speed, o1);
            k0.max_depth = get(P.max_depth, o1);
            if (P.horton) k0.g = at(P.cell, o1);
            if (raining) k0.rain_time = get(P.rain_time, o1);
            if (horton) { k0.f0 = at(P.f0, o1); k0.fc = at(P.fc, o1); k0.k = at(P.k, o1); }
        }
        hm = hn; zm = z0; lm = l0;
        h0 = h1; z0 = z1; l0 = l1; r0 = r1;
        h1 = h2; z1 = z2; l1 = l2; r1 = r2;
        h2 = h3; z2 = z3; l2 = l3;
        xs = xs3; ns = ns3; xw = xw2; nw = nw2;
        b1 = b2;
        qs1 = qs2; qw0 = qw1; d0 = d1; fs0 = fs1;
        o1 += row; o2 += row;
    }
}

// One step of the lattice form (solver_compact.py:439-641) but the CFL of
// the sides on strip and chunk edges, which k_lattice_close takes.
//
// A warp owns a strip of 32 lattice columns and P.rows rows and marches up
// it one row per iteration, the rows it needs held in registers and the
// west/east neighbours taken by shuffles. Iteration y forms q* of the south
// faces of row y + 2 and the west faces of row y + 1 (439-486), the donor
// factors of row y + 1 (491-514), the final discharge of the south faces
// of row y + 1 and the west faces of row y (516-522), the update of row y
// (525-610) and the CFL candidates (617-641) of row y's west and south
// sides whose cells this warp updated; and it loads what iteration y + 1
// will need (row y + 3 and the side discharges and Manning n first, the
// update inputs of row y + 1 after the update), so the loads of a row are
// in flight while the row before it is computed. Lanes 2..29 own the
// strip's 28 columns; lanes 0, 1, 30 and 31 are the halo the donor factors
// need. The first three iterations, below the chunk's rows, only fill the
// registers. No shared memory and no block barrier: each warp writes its
// counters and CFL minimum for the close pass and leaves. kParity: the buffer
// the step reads, which is the step's number in the batch (a batch starts on
// buffer 0 and a step that does nothing is followed by none that does), so the
// array bases are kernel parameters.
//
// Bound by instruction issue and memory latency (2048 x 1531 with Horton soil,
// 170 us: 59 % of active cycles issue with 21 of 64 warps, 24 by its 80 registers
// with 44 bytes of spills; DRAM at 20 %): 31 warp instructions per cell, 37
// before the inner path without liveness, boundaries and exterior sides (lattice_rows),
// 32-bit offsets on constant bases, rain rates instead of pixels and the rows
// that stay dry skipped. With the close pass that reduces a budget block per
// warp instead of per thread block (48 to 21 us at 2048 x 1531 with Horton
// soil), 32 steps: 4096 x 4096 dam break 25.0 to 16.9 ms, 2048 x 1531 7.95 to
// 6.29, 1003 x 741 2.85 (tiles) to 2.06.
template <int kMinBlocks, int kParity>
__global__ void __launch_bounds__(kNT, kMinBlocks) k_lattice_march(const __grid_constant__ Dev d)
{
    constexpr unsigned kAll = 0xffffffffu;
    const LatticePlan &P = d.lat;
    if (!d.ctl->active) return;
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int strip = blockIdx.x * warps + (threadIdx.x >> 5);
    if (strip >= P.strips) return;
    // limited cells, limited faces and wet cells of this lane, 10 bits each
    // (at most 2 x 256 rows), and the smallest donor factor's bits
    uint32_t counts = 0, min_bits = __float_as_uint(1.0f);
    unsigned long long best = kCflEmpty;
    const size_t w = (size_t)blockIdx.y * P.strips + strip, W = (size_t)P.strips * P.chunks;
    if (__ldg(P.plain + w)) lattice_rows<kParity, true>(d, strip, blockIdx.y, counts, min_bits, best);
    else lattice_rows<kParity, false>(d, strip, blockIdx.y, counts, min_bits, best);
    // counters and the CFL candidate of the warp, for the close pass: no
    // block barrier, so a warp leaves as soon as its strip is done
    const uint32_t n_lim = __reduce_add_sync(kAll, counts & 1023u);
    const uint32_t n_faces = __reduce_add_sync(kAll, (counts >> 10) & 1023u);
    const uint32_t n_wet = __reduce_add_sync(kAll, counts >> 20);
    min_bits = __reduce_min_sync(kAll, min_bits);
    best = warp_min_key(best);
    if (lane == 0) {
        P.part[w] = n_lim;
        P.part[W + w] = n_faces;
        P.part[2 * W + w] = n_wet;
        P.part[3 * W + w] = min_bits;
        P.part_cfl[w] = best;
    }
}

// After the march: the budget blocks the step touched (the canonical
// 256-cell tree of each term a block holds, device_budget.py:28-84, added
// into the compensated partials; scratch and marks cleared), the CFL
// candidates (solver_compact.py:617-641) of the sides on strip and chunk
// edges, whose two cells two different warps updated, and in the last block
// to finish the commit of the step and the prepare of the next.
__global__ void __launch_bounds__(256, 6) k_lattice_close(const __grid_constant__ Dev d)
{
    __shared__ unsigned long long sh_min[8];
    __shared__ uint32_t sh_cnt[8][4];
    __shared__ int last;
    const LatticePlan &P = d.lat;
    const nhf_mesh &m = d.m;
    Ctl *c = d.ctl;
    const int tid = threadIdx.x;
    const size_t e = (size_t)m.e_num;
    const int T = d.terms;
    // the last block's first thread looks at the dry key's own side (a value that
    // is not a number has no finite discharge)
    const int dry_side = blockIdx.x == gridDim.x - 1 && tid == 0 ? (int)(uint32_t)c->dry_key : -1;
    const int dry_at = dry_side > 0 ? P.gside[dry_side] : 0;
    // a warp looks at an even share of the budget blocks' marks, 32 at most at a
    // time, and takes the marked ones: lane l holds the tree's slots l, l + 32, .. l + 224, so the strides 128, 64 and
    // 32 are its own sums and a shuffle tree does 16 .. 1
    const int lane = tid & 31, warps = (int)gridDim.x * 8, per = min(32, (d.blocks + warps - 1) / warps);
    for (int base = per * ((int)blockIdx.x * 8 + (tid >> 5)); base < d.blocks; base += per * warps) {
        const int mine = base + lane;
        uint32_t mask = 0;
        if (lane < per && mine < d.blocks) {
            mask = P.touched[mine];
            if (mask) P.touched[mine] = 0u;
            if (P.touched_rain[mine]) { mask |= 1u; P.touched_rain[mine] = 0; }
        }
        for (uint32_t left = __ballot_sync(0xffffffffu, mask != 0u); left; left &= left - 1) {
            const int src = __ffs(left) - 1, b = base + src;
            for (uint32_t rest = __shfl_sync(0xffffffffu, mask, src); rest; rest &= rest - 1) {
                const int t = __ffs(rest) - 1;
                float *slot = P.terms + t * e + (size_t)b * 256 + lane;
                float v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = b * 256 + lane + 32 * k < m.e_num ? slot[32 * k] : 0.0f;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (v[k] != 0.0f) slot[32 * k] = 0.0f;
                double sum = (((double)v[0] + v[4]) + ((double)v[2] + v[6])) + (((double)v[1] + v[5]) + ((double)v[3] + v[7]));
                for (int stride = 16; stride >= 1; stride >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, stride);
                if (lane == 0) acc_add(d.acc_sum + (size_t)b * T + t, d.acc_comp + (size_t)b * T + t, sum);
            }
        }
    }
    const int active = c->active;
    unsigned long long best = kCflEmpty;
    uint32_t lim = 0, faces = 0, wet = 0, mb = __float_as_uint(1.0f);
    if (active) {
        // the march's per-warp counters and CFL minima
        const int W = P.strips * P.chunks;
        for (int w = blockIdx.x * 256 + tid; w < W; w += gridDim.x * 256) {
            lim += P.part[w];
            faces += P.part[W + w];
            wet += P.part[2 * W + w];
            mb = P.part[3 * W + w] < mb ? P.part[3 * W + w] : mb;
            best = P.part_cfl[w] < best ? P.part_cfl[w] : best;
        }
        const int p = c->parity ^ 1;  // the state the march just wrote
        const real dry_q = dry_side > 0 ? ((dry_at & 1) ? P.qh[p] : P.qv[p])[dry_at >> 1] : RC(0);
        const real *h = P.h[p], *qh = P.qh[p];
        const size_t lx = (size_t)P.lx;
        // counts below 2^31: the planner keeps the lattice under 2^30 points
        const int rows = P.chunks * P.rows, cols = P.strips * kOut;
        const int n_west = P.strips * rows, n = n_west + P.chunks * cols;
        for (int i = blockIdx.x * 256 + tid; i < n; i += gridDim.x * 256) {
            if (i < n_west) {  // west side of the first column of a strip, from the march's edge records
                const int s = i / rows, y = i % rows;
                if (s == 0) continue;  // west of strip 0: the border
                const float4 r = P.edge_first[i];
                const float2 l = P.edge_last[i - rows];
                if (r.w != 0.0f && l.x >= 0.0f) {
                    const size_t L = (size_t)(y + 2) * lx + (size_t)(s * kOut + 2);
                    lattice_cfl(d, P.len_v, r.z, l.y, l.x, r.y, r.x, P.side_v, (uint32_t)(4 * L), best);
                }
            } else {  // south side of the first row of a chunk
                const int k = i - n_west, ch = k / cols, x = 2 + k % cols;
                const size_t L = (size_t)(2 + ch * P.rows) * lx + (size_t)x;
                if (P.live[L] && P.live[L - lx])
                    lattice_cfl(d, P.len_h, qh[L], P.z[L - lx], h[L - lx], P.z[L], h[L], P.side_h, (uint32_t)(4 * L),
                                best);
            }
        }
        if (!(fabs(dry_q) < __uint_as_float(0x7f800000u))) note_cfl_nan(c);
    }
    best = warp_min_u64(best);
    lim = __reduce_add_sync(0xffffffffu, lim);
    faces = __reduce_add_sync(0xffffffffu, faces);
    wet = __reduce_add_sync(0xffffffffu, wet);
    mb = __reduce_min_sync(0xffffffffu, mb);
    if ((tid & 31) == 0) {
        sh_min[tid >> 5] = best;
        sh_cnt[tid >> 5][0] = lim; sh_cnt[tid >> 5][1] = faces; sh_cnt[tid >> 5][2] = wet; sh_cnt[tid >> 5][3] = mb;
    }
    __syncthreads();
    if (tid == 0) {
        unsigned long long bmin = kCflEmpty;
        uint32_t l = 0, f = 0, wt = 0, m2 = __float_as_uint(1.0f);
        for (int w = 0; w < 8; ++w) {
            bmin = sh_min[w] < bmin ? sh_min[w] : bmin;
            l += sh_cnt[w][0]; f += sh_cnt[w][1]; wt += sh_cnt[w][2];
            m2 = sh_cnt[w][3] < m2 ? sh_cnt[w][3] : m2;
        }
        if (bmin != kCflEmpty) atomicMin(&c->cfl_packed, bmin);
        if (l) {
            atomicAdd(&c->limited_cells, l);
            atomicMin(&c->min_scale_bits, m2);
        }
        if (f) atomicAdd(&c->limited_faces, f);
        if (wt) atomicAdd(&c->wet, wt);
        __threadfence();
        const unsigned ticket = atomicAdd(&c->done_blocks, 1u);
        last = last_of(ticket, gridDim.x);
    }
    __syncthreads();
    if (!last) return;
    if (last == 2) rescan_cfl(d, LatticeState{&P, c->parity ^ 1});
    if (tid != 0) return;
    __threadfence();
    c->done_blocks = 0;
    if (active) {
        set_cfl(c, last == 2);
        c->parity ^= 1;
    }
    finish_step(c);
    if (c->slot < d.batch_size) lattice_prepare(d, c);
}

// Static lattice arrays from the caller's mesh (once).
__global__ void k_lattice_setup(const __grid_constant__ Dev d)
{
    const LatticePlan &P = d.lat;
    const nhf_mesh &m = d.m;
    const size_t n = (size_t)P.lx * P.ly;
    for (size_t L = (size_t)blockIdx.x * blockDim.x + threadIdx.x; L < n; L += (size_t)gridDim.x * blockDim.x) {
        const int g = P.cell[L];
        P.bi[L] = (int16_t)(g ? m.boundary_id[g] : -1);
        if (P.horton) {
            P.f0[L] = g ? m.f0[g] : RC(0);
            P.fc[L] = g ? m.fc[g] : RC(0);
            P.k[L] = g ? m.k[g] : RC(0);
        }
        const int sv = P.side_v[L], sh = P.side_h[L];
        P.nv[L] = sv ? m.side_n[sv] : RC(0);
        P.nh[L] = sh ? m.side_n[sh] : RC(0);
    }
}

// Batch start: the caller's state into lattice order (buffer 0).
__global__ void k_lattice_gather(const __grid_constant__ Dev d)
{
    const LatticePlan &P = d.lat;
    const nhf_mesh &m = d.m;
    const size_t n = (size_t)P.lx * P.ly;
    const bool raining = P.rain_cells && d.ctl->raining != 0;
    for (size_t L = (size_t)blockIdx.x * blockDim.x + threadIdx.x; L < n; L += (size_t)gridDim.x * blockDim.x) {
        const int g = P.cell[L];
        if (raining) P.rate[L] = g ? d.rain_rates[m.rain_index[g]] : RC(0);  // fixed during a batch
        P.h[0][L] = m.depth[g];  // holes and the border hold the sentinel's values
        if (!g) P.h[1][L] = m.depth[0];
        P.z[L] = m.bed[g];
        if (g) {
            P.rain_time[L] = m.rain_time[g];
            P.infil[L] = m.infiltration[g];
            P.max_depth[L] = m.max_depth[g];
            P.max_speed[L] = m.max_speed[g];
            // extrema below zero would rise to a dry cell's zero, and infiltration
            // below zero would wet it: no idle rows then
            if (m.max_depth[g] < RC(0) || m.max_speed[g] < RC(0) || !(m.infiltration[g] >= RC(0))) *P.odd = 1;
            P.peak_hi[L] = m.peak_hi[g];
            P.peak_lo[L] = m.peak_lo[g];
        }
        const int sv = P.side_v[L], sh = P.side_h[L];
        P.qv[0][L] = sv ? m.q[sv] : RC(0);
        P.qh[0][L] = sh ? m.q[sh] : RC(0);
    }
}

// Batch end: the lattice state back into the caller's arrays.
__global__ void k_lattice_scatter(const __grid_constant__ Dev d)
{
    __shared__ bool last;
    const LatticePlan &P = d.lat;
    const nhf_mesh &m = d.m;
    Ctl *c = d.ctl;
    const int p = c->parity;
    const size_t n = (size_t)P.lx * P.ly;
    for (size_t L = (size_t)blockIdx.x * blockDim.x + threadIdx.x; L < n; L += (size_t)gridDim.x * blockDim.x) {
        const int g = P.cell[L];
        if (g) {
            m.depth[g] = P.h[p][L];
            m.rain_time[g] = P.rain_time[L];
            m.infiltration[g] = P.infil[L];
            m.max_depth[g] = P.max_depth[L];
            m.max_speed[g] = P.max_speed[L];
            m.peak_hi[g] = P.peak_hi[L];
            m.peak_lo[g] = P.peak_lo[L];
        }
        const int sv = P.side_v[L], sh = P.side_h[L];
        if (sv) m.q[sv] = P.qv[p][L];
        if (sh) m.q[sh] = P.qh[p][L];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned ticket = atomicAdd(&c->done_blocks, 1u);
        last = ticket == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        c->done_blocks = 0;
        c->parity = 0;
        *P.odd = 0;
    }
}

// Which warps' cells are all live and off the boundaries (once): a warp per
// strip and chunk looks at every row its march loads.
__global__ void k_lattice_plain(const __grid_constant__ Dev d)
{
    const LatticePlan &P = d.lat;
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= P.strips * P.chunks) return;
    const int strip = w % P.strips, y0 = 2 + (w / P.strips) * P.rows;
    bool plain = true;
    for (int y = y0 - 2; y < y0 + P.rows + 3; ++y) {
        const size_t L = (size_t)y * P.lx + (size_t)(strip * kOut + lane);
        plain = plain && P.live[L] && P.bi[L] < 0;
    }
    plain = __all_sync(0xffffffffu, plain);
    if (lane == 0) P.plain[w] = plain ? 1 : 0;
}

int stream_grid(size_t n)
{
    size_t g = (n + 255) / 256;
    return (int)std::min<size_t>(std::max<size_t>(g, 1), 148 * 16);
}

}  // namespace

// ------------------------------------------------------------------ planner

// Rows per chunk, warps per block and resident warps per SM of the march.
// A warp marches its rows after three rows of warm-up: more rows waste less
// on those, fewer rows finish more evenly and, below one wave of blocks, give
// idle SMs work. Measured (us per 32 steps by rows): 4096 x 4096 dam break 12:
// 17198, 16: 17053, 24: 17462; 2048 x 2048 8: 5734, 16: 6219; 1003 x 741 4: 2141,
// 8: 2043, 10: 2230; 600 x 600 4: 1425, 8: 1861; 421 x 307 2: 1037, 4: 1242. So 16
// rows from four waves on, else 8, halved while blocks fill less than 9/10 of
// the chip. 24 resident warps per SM (80 registers) beat 32 (64 registers,
// 170 bytes of spills): 2048 x 1531 6104 against 6187 us, 1003 x 741 2047 against
// 2270, 4096 x 4096 16905 against 17160. NHF_LATTICE_ROWS, NHF_LATTICE_WARPS
// (warps per block, 1..8) and NHF_LATTICE_BLOCKS (2, 3 or 4: 512, 768 or
// 1024 resident threads per SM, the register budget) override the choice.
static void lattice_shape(LatticePlan *P)
{
    // warps leave independently (no block barrier): small blocks free their
    // slots as soon as their strips are done
    const char *bw = getenv("NHF_LATTICE_WARPS");
    const int warps = (bw && atoi(bw) >= 1 && atoi(bw) <= kWarps) ? atoi(bw) : 2;
    const int per_row = (P->strips + warps - 1) / warps;  // blocks across the strips
    P->block_warps = (P->strips + per_row - 1) / per_row;  // <= warps, as even as the strips allow
    const char *occ = getenv("NHF_LATTICE_BLOCKS");
    const int want = occ ? atoi(occ) : 0;
    P->min_blocks = (want >= 2 && want <= 4) ? want : 3;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        sms = 148;
    }
    const long long wave = (long long)sms * P->min_blocks * kWarps / P->block_warps;  // resident blocks
    const int need = P->ny + 1;
    auto blocks = [&](int rows) { return (long long)((need + rows - 1) / rows) * per_row; };
    int rows = blocks(16) >= 4 * wave ? 16 : 8;
    while (rows > 2 && 10 * blocks(rows) < 9 * wave) rows /= 2;
    const char *env = getenv("NHF_LATTICE_ROWS");
    if (env && atoi(env) >= 1 && atoi(env) <= 256) rows = atoi(env);  // a lane's counters hold 10 bits
    P->rows = rows;
    P->chunks = (need + rows - 1) / rows;
}

int lattice_build(const Dev &d, cudaStream_t st, LatticeBuild *out, char *why, size_t why_len)
{
    const nhf_mesh &m = d.m;
    auto no = [&](const char *msg) { snprintf(why, why_len, "%s", msg); return 1; };
    const int e = m.e_num, s = m.s_num;
    if (e < 1 + 1024) return no("fewer than 1024 cells");
    if (!d.theta_one) return no("theta < 1");
    if (m.hang_cells > 0) return no("hanging edges");
    if (d.terms > 32) return no("more than four boundaries");
    if (m.isl_len != 4 * (e - 1)) return no("not one side per face");
    std::vector<float> x(e), y(e), w(e), hg(e), area(e), len(s);
    std::vector<int32_t> topo((size_t)s * 3), fptr((size_t)e * 4), fcnt((size_t)e * 4), isl(m.isl_len);
    if (cudaMemcpyAsync(x.data(), m.x, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(y.data(), m.y, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(w.data(), m.width, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(hg.data(), m.height, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(area.data(), m.area, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(len.data(), m.length, 4 * (size_t)s, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(topo.data(), m.topology, 12 * (size_t)s, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(fptr.data(), m.face_ptr, 16 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(fcnt.data(), m.face_count, 16 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(isl.data(), m.isl_data, 4 * (size_t)m.isl_len, cudaMemcpyDeviceToHost, st) ||
        cudaStreamSynchronize(st))
        return no("copy of the mesh tables failed");
    const float W = w[1], H = hg[1], A = area[1];
    float x0 = x[1], y0 = y[1];
    for (int c = 1; c < e; ++c) {
        if (w[c] != W || hg[c] != H || area[c] != A) return no("cell sizes differ");
        x0 = std::min(x0, x[c]);
        y0 = std::min(y0, y[c]);
        for (int dd = 0; dd < 4; ++dd)
            if (fcnt[4 * c + dd] != 1) return no("a face without exactly one side");
    }
    if (!(W > 0.0f) || !(H > 0.0f)) return no("empty cells");
    std::vector<int32_t> ci(e), cj(e);
    int nx = 0, ny = 0;
    for (int c = 1; c < e; ++c) {
        const double fi = ((double)x[c] - x0) / W, fj = ((double)y[c] - y0) / H;
        const long long i = llround(fi), j = llround(fj);
        if (std::fabs(fi - i) > 1e-3 || std::fabs(fj - j) > 1e-3 || i > (1 << 20) || j > (1 << 20))
            return no("cell centres off a lattice");
        ci[c] = (int)i; cj[c] = (int)j;
        nx = std::max(nx, (int)i + 1);
        ny = std::max(ny, (int)j + 1);
    }
    if ((double)nx * ny > 1.5 * (e - 1)) return no("lattice mostly empty");
    LatticePlan P{};
    P.nx = nx; P.ny = ny;
    // strips of 28 columns cover cell columns 0..nx (column nx: the east
    // sides), chunks of P.rows rows cover cell rows 0..ny
    P.strips = (nx + 1 + kOut - 1) / kOut;
    lattice_shape(&P);
    P.lx = P.strips * kOut + kWest + 2;
    P.ly = P.chunks * P.rows + 5;  // 2 rows below, 3 above: the march loads a row ahead
    const size_t nl = (size_t)P.lx * P.ly;
    if (nl >= ((size_t)1 << 30)) return no("lattice too large");
    auto at = [&](int i, int j) { return (size_t)(j + 2) * P.lx + (i + kWest); };
    std::vector<int32_t> cell(nl, 0), side_v(nl, 0), side_h(nl, 0), glat(e, 0), gside(s, 0);
    std::vector<uint8_t> live(nl, 0);
    for (int c = 1; c < e; ++c) {
        const size_t L = at(ci[c], cj[c]);
        if (cell[L]) return no("two cells at one lattice point");
        cell[L] = c; live[L] = 1; glat[c] = (int32_t)L;
    }
    auto cell_at = [&](int i, int j) -> int {
        if (i < 0 || j < 0 || i >= nx || j >= ny) return 0;
        return cell[at(i, j)];
    };
    // every face's side joins the lattice neighbours (west/east: orientation
    // 2, lower = west; south/north: orientation 1, lower = south)
    bool have_v = false, have_h = false;
    float sdc_v = 0.0f, sdc_h = 0.0f, len_v = 0.0f, len_h = 0.0f;
    std::vector<int> seen(s, 0);
    for (int c = 1; c < e; ++c) {
        const int i = ci[c], j = cj[c];
        const int nb[4] = {cell_at(i - 1, j), cell_at(i + 1, j), cell_at(i, j - 1), cell_at(i, j + 1)};
        for (int dd = 0; dd < 4; ++dd) {
            const int p = fptr[4 * c + dd];
            if (p < 0 || p >= m.isl_len) return no("a face pointer outside the side list");
            const int sid = isl[p];
            if (sid < 1 || sid >= s) return no("a face lists an invalid side");
            const int so = topo[3 * sid], lo = topo[3 * sid + 1], hi = topo[3 * sid + 2];
            const bool vertical = dd < 2;
            const int want_lo = (dd == 0 || dd == 2) ? nb[dd] : c, want_hi = (dd == 0 || dd == 2) ? c : nb[dd];
            if (so != (vertical ? 2 : 1) || lo != want_lo || hi != want_hi) return no("sides off the lattice");
            // the lattice side is the west / south face of its higher cell
            // (or of the lattice point east / north of its lower cell)
            const size_t L = (dd == 0 || dd == 2) ? at(i, j) : (dd == 1 ? at(i + 1, j) : at(i, j + 1));
            std::vector<int32_t> &map = vertical ? side_v : side_h;
            if (map[L] && map[L] != sid) return no("two sides at one lattice face");
            map[L] = sid;
            gside[sid] = (int32_t)((L << 1) | (vertical ? 0u : 1u));
            seen[sid] = 1;
            const float l = len[sid];
            if (vertical) {
                if (have_v && l != len_v) return no("side lengths differ");
                len_v = l;
            } else {
                if (have_h && l != len_h) return no("side lengths differ");
                len_h = l;
            }
            if (lo && hi) {  // interior: centre distance as k_initialize computes it
                const float dist = vertical ? std::max(std::fabs(x[hi] - x[lo]), 0.01f)
                                           : std::max(std::fabs(y[hi] - y[lo]), 0.01f);
                float &ref = vertical ? sdc_v : sdc_h;
                bool &have = vertical ? have_v : have_h;
                if (have && dist != ref) return no("centre distances differ");
                ref = dist;
                have = true;
            }
        }
    }
    for (int sid = 1; sid < s; ++sid)
        if (!seen[sid]) return no("a side no face lists");
    if (!have_v || !have_h) return no("no interior side in one direction");
    P.sdc_v = sdc_v; P.sdc_h = sdc_h; P.len_v = len_v; P.len_h = len_h;
    P.area = A; P.width = W; P.height = H;
    auto inverse = [](float b) {   // 1 / b where b is a power of two, else 0
        int e;
        return std::frexp(b, &e) == 0.5f && e > -100 && e < 100 ? 1.0f / b : 0.0f;
    };
    P.inv_sdc_v = inverse(sdc_v); P.inv_sdc_h = inverse(sdc_h); P.inv_area = inverse(A);
    // rain pixels and Horton parameters per lattice cell only when they vary
    std::vector<int32_t> rain(e);
    std::vector<float> f0(e), fc(e), kk(e);
    if (cudaMemcpyAsync(rain.data(), m.rain_index, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(f0.data(), m.f0, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(fc.data(), m.fc, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) ||
        cudaMemcpyAsync(kk.data(), m.k, 4 * (size_t)e, cudaMemcpyDeviceToHost, st) || cudaStreamSynchronize(st))
        return no("copy of the cell parameters failed");
    P.rain_cells = 0;
    P.horton = 0;
    for (int c = 1; c < e; ++c) {
        if (rain[c] != 0) P.rain_cells = 1;
        if (f0[c] != 0.0f || fc[c] != 0.0f || kk[c] != 0.0f) P.horton = 1;
    }
    // device memory: maps, state copies, static arrays, budget scratch
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 255) & ~size_t(255); return o; };
    const size_t o_cell = take(4 * nl), o_sv = take(4 * nl), o_sh = take(4 * nl), o_live = take(nl);
    const size_t o_glat = take(4 * (size_t)e), o_gside = take(4 * (size_t)s);
    size_t o_h[2], o_qv[2], o_qh[2];
    for (int k = 0; k < 2; ++k) { o_h[k] = take(4 * nl); o_qv[k] = take(4 * nl); o_qh[k] = take(4 * nl); }
    const size_t o_z = take(4 * nl), o_nv = take(4 * nl), o_nh = take(4 * nl), o_bi = take(2 * nl);
    const size_t o_rain = P.rain_cells ? take(4 * nl) : 0;
    const size_t o_rt = take(4 * nl), o_inf = take(4 * nl), o_md = take(4 * nl), o_ms = take(4 * nl);
    const size_t o_ph = take(4 * nl), o_pl = take(4 * nl);
    size_t o_f0 = 0, o_fc = 0, o_k = 0;
    if (P.horton) { o_f0 = take(4 * nl); o_fc = take(4 * nl); o_k = take(4 * nl); }
    const size_t o_terms = take(4 * (size_t)d.terms * e), o_touch = take(4 * (size_t)d.blocks);
    const size_t o_touch0 = take(d.blocks), o_odd = take(4);
    const size_t n_warps = (size_t)P.strips * P.chunks;
    const size_t o_plain = take(n_warps);
    const size_t o_part = take(16 * n_warps), o_pcfl = take(8 * n_warps);
    const size_t n_edge = (size_t)P.strips * P.chunks * P.rows;
    const size_t o_efirst = take(16 * n_edge), o_elast = take(8 * n_edge);
    char *mem = nullptr;
    if (cudaMalloc((void **)&mem, off)) { cudaGetLastError(); return no("no device memory for the lattice"); }
    out->device_memory = mem;
    if (cudaMemsetAsync(mem, 0, off, st) ||
        cudaMemcpyAsync(mem + o_cell, cell.data(), 4 * nl, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(mem + o_sv, side_v.data(), 4 * nl, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(mem + o_sh, side_h.data(), 4 * nl, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(mem + o_live, live.data(), nl, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(mem + o_glat, glat.data(), 4 * (size_t)e, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(mem + o_gside, gside.data(), 4 * (size_t)s, cudaMemcpyHostToDevice, st) ||
        cudaStreamSynchronize(st))
        return no("upload of the lattice maps failed");
    P.cell = (const int32_t *)(mem + o_cell);
    P.side_v = (const int32_t *)(mem + o_sv);
    P.side_h = (const int32_t *)(mem + o_sh);
    P.live = (const uint8_t *)(mem + o_live);
    P.glat = (const int32_t *)(mem + o_glat);
    P.gside = (const int32_t *)(mem + o_gside);
    for (int k = 0; k < 2; ++k) {
        P.h[k] = (real *)(mem + o_h[k]);
        P.qv[k] = (real *)(mem + o_qv[k]);
        P.qh[k] = (real *)(mem + o_qh[k]);
    }
    P.z = (real *)(mem + o_z); P.nv = (real *)(mem + o_nv); P.nh = (real *)(mem + o_nh);
    P.bi = (int16_t *)(mem + o_bi);
    P.rate = P.rain_cells ? (real *)(mem + o_rain) : nullptr;
    P.rain_time = (real *)(mem + o_rt); P.infil = (real *)(mem + o_inf);
    P.max_depth = (real *)(mem + o_md); P.max_speed = (real *)(mem + o_ms);
    P.peak_hi = (uint32_t *)(mem + o_ph); P.peak_lo = (uint32_t *)(mem + o_pl);
    if (P.horton) { P.f0 = (real *)(mem + o_f0); P.fc = (real *)(mem + o_fc); P.k = (real *)(mem + o_k); }
    P.terms = (float *)(mem + o_terms);
    P.touched = (uint32_t *)(mem + o_touch);
    P.touched_rain = (uint8_t *)(mem + o_touch0);
    P.odd = (int32_t *)(mem + o_odd);
    P.plain = (uint8_t *)(mem + o_plain);
    P.part = (uint32_t *)(mem + o_part);
    P.part_cfl = (unsigned long long *)(mem + o_pcfl);
    P.edge_first = (float4 *)(mem + o_efirst);
    P.edge_last = (float2 *)(mem + o_elast);
    Dev dd = d;
    dd.lat = P;
    k_lattice_setup<<<stream_grid(nl), 256, 0, st>>>(dd);
    k_lattice_plain<<<(P.strips * P.chunks + 7) / 8, 256, 0, st>>>(dd);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st)) return no("lattice setup failed");
    out->plan = P;
    return 0;
}

void lattice_enqueue_batch_start(const Dev &d, cudaStream_t s)
{
    k_lattice_gather<<<stream_grid((size_t)d.lat.lx * d.lat.ly), 256, 0, s>>>(d);
}

template <int kMinBlocks>
static void launch_march(const Dev &d, const dim3 &grid, const dim3 &block, int parity, cudaStream_t s)
{
    if (parity) k_lattice_march<kMinBlocks, 1><<<grid, block, 0, s>>>(d);
    else k_lattice_march<kMinBlocks, 0><<<grid, block, 0, s>>>(d);
}

void lattice_enqueue_step(const Dev &d, int step, cudaStream_t s)
{
    const LatticePlan &P = d.lat;
    const int per_block = (P.strips + P.block_warps - 1) / P.block_warps;
    const dim3 grid(per_block, P.chunks), block(32 * P.block_warps);
    if (P.min_blocks == 2) launch_march<2>(d, grid, block, step & 1, s);
    else if (P.min_blocks == 3) launch_march<3>(d, grid, block, step & 1, s);
    else launch_march<4>(d, grid, block, step & 1, s);
    const long long edges = (long long)P.strips * P.chunks * (P.rows + kOut);
    const long long work = std::max<long long>(edges / 256, d.blocks / 8);
    k_lattice_close<<<(int)std::max<long long>(1, std::min<long long>(148 * 8, work)), 256, 0, s>>>(d);
}

void lattice_enqueue_batch_end(const Dev &d, cudaStream_t s)
{
    k_lattice_scatter<<<stream_grid((size_t)d.lat.lx * d.lat.ly), 256, 0, s>>>(d);
    tiled_enqueue_velocity(d, s);
}

}  // namespace nhf

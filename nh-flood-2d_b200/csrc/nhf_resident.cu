// The resident form of the fused tiled step: a whole batch in one cooperative
// launch, for meshes whose tiles all fit the GPU at once.
//
// On such meshes a step of one launch is latency, not work: 256 x 256 cells
// took 21 us per step and 83 x 61 cells 20 us, most of it the launch, the copy
// of the tile's tables, and the last block's serial commit. Here a block keeps
// its tile for the whole batch: index tables, bed, lengths, Manning n and the
// state of the tile and its rings stay in shared memory, the extrema in
// registers. A step is the fused-CFL form of nhf_tiled.cu (three rings, the
// same expressions, so the same bits): momentum of the faces of rings <= 2,
// donor factors of rings <= 2, final discharge of the faces of rings <= 1,
// depth of rings <= 1, CFL of the owned sides. Rings 0 and 1 then hold their
// new state already; the blocks exchange the depth of rings 2 and 3 and the
// discharge of the outer faces.
//
// The exchange needs no fence and no barrier. Each exchanged value is one
// 64-bit word, the F32 bits and the number of the step they belong to, written
// and read whole; a reader polls the word until it carries its step. The CFL
// minimum travels the same way: each block writes its smallest (CFL bits, side
// id) key with a phase bit, the first warp of every block reads all blocks'
// keys, takes the minimum and runs the clock (StepClock.choose) for its block,
// so no result travels back, while the other warps collect the outer rings and
// reduce budget terms. Having everyone's key of step s also says that everyone
// has read the words of step s - 1, so two buffers of words suffice. The grid
// is launched cooperatively (all blocks resident at once). A wait gives up after
// kSpinLimit reads (NHF_RESIDENT_SPINS in the environment at nhf_initialize
// sets another limit), its thread waits for nothing more and its block leaves;
// the others' waits for that block run out in turn. The batch is void then, its
// first trace row says NHF_STEP_STALLED, and so do later batches until
// nhf_initialize.
//
// Measured, one batch of 32 steps end to end, against a launch per step:
// 83 x 61 cells 646 to 271 us, 256 x 256 682 to 352, 421 x 307 numbered by
// rows 1007 to 546, quadtrees of 16,584 cells 783 to 339, 0.19 M 1343 to 723,
// 0.11 M with theta = 0.7 1133 to 659. What is left of a step of 7 us (83 x 61)
// is four fifths latency: seven block-wide phases and one exchange through L2
// (about 2,500 cycles from a block's key to the last block's reading it);
// schedulers issue in 41 % of cycles.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "nhf_common.cuh"
#include "nhf_math.cuh"

namespace nhf {
namespace {

typedef unsigned long long u64;

constexpr int kSpinLimit = 1 << 22;      // reads of a word before a wait gives up (seconds)
constexpr u64 kPhase = 1ULL << 63;
constexpr int kMaxBoundaries = 4;
constexpr int kMaxKeys = 5;              // keys a lane of the first warp reads: grids of up to 160 blocks
// A local side is its lower and higher slot (14 bits each) and flags: its level
// difference takes hanging gradients, it is vertical, its discharge is exchanged,
// an open face lies beyond it (theta < 1).
constexpr uint32_t kSlot = 0x3fffu, kHangSide = 0x4000u, kVertical = 0x8000u, kShared = 0x80000000u,
                   kOpen = 0x40000000u;

__device__ __forceinline__ void put_word(u64 *p, u64 v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ u64 get_word(const u64 *p)
{
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ u64 value_word(float v, uint32_t step) { return ((u64)step << 32) | __float_as_uint(v); }

// The value of step `step` at p, given a first read w of it.
__device__ __forceinline__ float await_value(const u64 *p, u64 w, uint32_t step, int limit, bool &lost)
{
    for (int spin = 0; (uint32_t)(w >> 32) != step && spin < limit && !lost; ++spin) w = get_word(p);
    lost = lost || (uint32_t)(w >> 32) != step;
    return __uint_as_float((uint32_t)w);
}

// The clock of a batch (the members of Ctl that StepClock works on), one copy
// per block.
struct Clock {
    uint32_t now[2], next[2], origin[2], step_end[2];
    float dt, local, end_local;
    int32_t active;
};

// A side at a resolution change: its local index, the gradients it takes (-1:
// none) with their offsets, and their values.
struct Hanging {
    int32_t j, item[2];
    real offset[2], value[2];
};

struct Sizes {
    size_t acc, hang, h, z, sc, area, rain, q, len, dx, n, lohi, nb, gid, stage, r1, faces, bi, total;
};

// Shared memory of one block, in bytes from its start. Sides have one more
// entry, of no length, which stands for the faces a cell does not have.
__host__ __device__ inline Sizes sizes_of(const ResidentArgs &r, int terms, bool theta_one, int per_face, int stage)
{
    Sizes s;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 15) & ~size_t(15); return o; };
    const int T = r.plan.tile, E = r.plan.max_ext, D = r.max_don + 1, S = r.plan.max_sides + 1;
    s.acc = take((size_t)(T / 256) * terms * 16);
    s.hang = take(sizeof(Hanging) * r.max_hang);
    s.h = take(4 * (size_t)E);
    s.z = take(4 * (size_t)E);
    s.sc = take(4 * (size_t)D);
    s.area = take(4 * (size_t)D);
    s.rain = take(4 * (size_t)D);
    s.q = take(4 * (size_t)S);
    s.len = take(4 * (size_t)S);
    s.dx = take(4 * (size_t)S);
    s.n = take(4 * (size_t)S);
    s.lohi = take(4 * (size_t)S);
    s.nb = take(theta_one ? 0 : 4 * (size_t)S);
    s.gid = take(4 * (size_t)r.max_owned);
    s.stage = take(4 * (size_t)stage * T);
    s.r1 = take(8 * (size_t)r.max_r1);
    s.faces = take(8 * (size_t)per_face * D);
    s.bi = take(2 * (size_t)D);
    s.total = off;
    return s;
}

// A cell's local sides, one or two per face (west, east, south, north).
template <bool kTwo>
struct Faces {
    uint32_t w[kTwo ? 4 : 2];
    __device__ __forceinline__ int side(int face, int k) const
    {
        const int e = kTwo ? 2 * face + k : face;
        return (int)((w[e >> 1] >> (16 * (e & 1))) & 0xffffu);
    }
};

template <bool kTwo>
__device__ __forceinline__ Faces<kTwo> faces_of(const unsigned char *table, int slot)
{
    Faces<kTwo> f;
    if constexpr (kTwo) {
        const uint4 v = reinterpret_cast<const uint4 *>(table)[slot];
        f.w[0] = v.x; f.w[1] = v.y; f.w[2] = v.z; f.w[3] = v.w;
    } else {
        const uint2 v = reinterpret_cast<const uint2 *>(table)[slot];
        f.w[0] = v.x; f.w[1] = v.y;
    }
    return f;
}

// prepare_step's snapshot of the limiting side (solver_compact.py:372-382). Each
// block keeps its own until the batch's end: the owner of the last one taken
// writes it out, so the control block's words have one writer and no order
// between blocks matters.
struct Limit {
    float value[5];
    int32_t id[3];
    int32_t mine;   // 1: the batch's last snapshot so far is this block's
};

// The snapshot of a batch's first step, from the caller's state.
__device__ __noinline__ void snapshot_limit(const Dev &d, float ndt, int si, Limit *out)
{
    const nhf_mesh &m = d.m;
    const int el = m.topology[3 * si + 1], eh = m.topology[3 * si + 2];
    const real h = flow_depth_of(m, m.depth, si);
    out->value[0] = ndt;
    out->value[1] = m.depth[el]; out->value[2] = m.depth[eh];
    out->value[3] = h;
    out->value[4] = m.q[si] / rmax(h, RC(1e-30));
    out->id[0] = si; out->id[1] = el; out->id[2] = eh;
    out->mine = 1;
}

template <bool kThetaOne, bool kTwo, int NT, int T>
__global__ void __launch_bounds__(NT, 1) k_resident(const __grid_constant__ Dev d, const __grid_constant__ ResidentArgs r)
{
    constexpr int CPT = (T + NT - 1) / NT;      // own cells per thread (the first T threads have one when NT > T)
    constexpr int kBlocks = T / 256;            // budget blocks of a tile
    constexpr int kWarps = NT / 32;
    constexpr int kStage = T >= 768 ? 1 : 2;    // budget terms reduced together
    constexpr unsigned kAll = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Clock ck;
    __shared__ float sh_coef[2 * kMaxBoundaries], sh_values[kMaxBoundaries], sh_levels[kMaxBoundaries];
    __shared__ int sh_kind[kMaxBoundaries];
    __shared__ u64 sh_best;   // the block's CFL bits << 32 | local side
    __shared__ uint32_t sh_cnt[3], sh_minbits, sh_near, sh_mask[kBlocks];
    __shared__ uint32_t sh_row[NHF_TRACE_COLS], sh_end[NHF_MAX_BATCH][2];
    __shared__ float sh_ndt;
    __shared__ int sh_arg, sh_slot, sh_hang, sh_last;
    __shared__ Limit sh_limit;

    const nhf_mesh &m = d.m;
    Ctl *c = d.ctl;
    const TilePlan &P = r.plan;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_blocks = gridDim.x;
    const int terms_n = d.terms, B = m.b_num;
    const Sizes at = sizes_of(r, terms_n, kThetaOne, kTwo ? 2 : 1, kStage);
    double *sh_acc = reinterpret_cast<double *>(smem_raw + at.acc);   // [block][term] {sum, compensation}
    Hanging *sh_hg = reinterpret_cast<Hanging *>(smem_raw + at.hang);
    float *sh_h = reinterpret_cast<float *>(smem_raw + at.h);
    float *sh_z = reinterpret_cast<float *>(smem_raw + at.z);
    float *sh_s = reinterpret_cast<float *>(smem_raw + at.sc);
    float *sh_area = reinterpret_cast<float *>(smem_raw + at.area);
    float *sh_rain = reinterpret_cast<float *>(smem_raw + at.rain);
    float *sh_q = reinterpret_cast<float *>(smem_raw + at.q);
    float *sh_len = reinterpret_cast<float *>(smem_raw + at.len);
    float *sh_dx = reinterpret_cast<float *>(smem_raw + at.dx);
    float *sh_n = reinterpret_cast<float *>(smem_raw + at.n);
    uint32_t *sh_lohi = reinterpret_cast<uint32_t *>(smem_raw + at.lohi);
    float *sh_nb = reinterpret_cast<float *>(smem_raw + at.nb);       // theta < 1: boundary_neighbor_sum
    int32_t *sh_gid = reinterpret_cast<int32_t *>(smem_raw + at.gid);  // owned sides
    float *sh_stage = reinterpret_cast<float *>(smem_raw + at.stage);
    float2 *sh_r1 = reinterpret_cast<float2 *>(smem_raw + at.r1);     // rain time, capacity of ring-1 cells
    unsigned char *sh_faces = smem_raw + at.faces;
    int16_t *sh_bi = reinterpret_cast<int16_t *>(smem_raw + at.bi);

    const int4 *head = P.tile_head + 4 * blockIdx.x;
    const int4 h0 = head[0], h1 = head[1], h2 = head[2], h3 = head[3];
    const int n_ext = h0.x, n_r0 = h0.y, n_r01 = h0.z, n_don = h0.w;
    const int n_sides = h1.x, n_owned = h1.y, n_qf = h1.z, r0off = h1.w;
    const int cbase = h2.y, sbase = h2.z;
    const int32_t *ext = P.ext_rel + h2.w, *srel = P.side_rel + h3.x;

    if (c->stalled) return;   // an earlier batch stalled: its words are out of step

    // ---- the tile, once per batch
    const int raining = c->raining;
    const uint32_t epoch0 = c->epoch;
    const uint32_t turn = c->batches & 1u;
    float limit0 = c->limit_value[0];   // the first warp's: the smallest CFL candidate snapshot so far
    if (tid == 0) {
        ck.now[0] = c->now[0]; ck.now[1] = c->now[1];
        ck.next[0] = r.words[0]; ck.next[1] = r.words[1];
        ck.origin[0] = r.words[2]; ck.origin[1] = r.words[3];
        sh_ndt = c->ndt; sh_arg = c->cfl_arg; sh_slot = 0; sh_hang = 0; sh_limit.mine = 0;
        sh_cnt[0] = sh_cnt[1] = sh_cnt[2] = 0u; sh_minbits = __float_as_uint(1.0f);
        sh_s[0] = 0.0f;  // donor factor of the exterior sentinel
        sh_q[n_sides] = sh_len[n_sides] = 0.0f;
    }
    if (tid < B) sh_kind[tid] = m.kind[tid];
    if (tid < 2 * B) sh_coef[tid] = d.coef[tid];
    if (blockIdx.x == 0)
        for (int i = tid; i < NHF_MAX_BATCH * NHF_TRACE_COLS; i += NT) c->trace[i] = 0u;
    for (int i = tid; i < kBlocks * terms_n; i += NT) {
        const int blk = (cbase >> 8) + i / terms_n;
        const size_t g = (size_t)blk * terms_n + i % terms_n;
        sh_acc[2 * i] = blk < d.blocks ? d.acc_sum[g] : 0.0;
        sh_acc[2 * i + 1] = blk < d.blocks ? d.acc_comp[g] : 0.0;
    }
    for (int i = tid; i < n_ext; i += NT) {
        const int g = i ? cbase + ext[i] : 0;
        sh_h[i] = m.depth[g];
        sh_z[i] = m.bed[g];
        if (i >= 1 && i <= n_don) {
            sh_area[i] = m.area[g];
            sh_bi[i] = (int16_t)m.boundary_id[g];
            sh_rain[i] = raining ? d.rain_rates[m.rain_index[g]] : 0.0f;
            const uint32_t fd = P.face_desc[h3.y + i];
            const uint16_t *fidx = P.face_idx + h3.z + (fd & 0xffffu);
            uint16_t *mine = reinterpret_cast<uint16_t *>(sh_faces) + (kTwo ? 8 : 4) * i;
            for (int dd = 0, p = 0; dd < 4; ++dd) {
                const int cnt = (int)((fd >> (16 + 4 * dd)) & 15u);
                for (int k = 0; k < (kTwo ? 2 : 1); ++k)
                    mine[(kTwo ? 2 : 1) * dd + k] = k < cnt ? fidx[p + k] : (uint16_t)n_sides;
                p += cnt;
            }
        }
        if (i > n_r0 && i <= n_r01) sh_r1[i - n_r0 - 1] = make_float2(m.rain_time[g], m.infiltration[g]);
    }
    __syncthreads();
    for (int j = tid; j < n_sides; j += NT) {
        const int gid = sbase + srel[j];
        const float2 sdn = d.sdn[gid];
        if (j < n_owned) sh_gid[j] = gid;
        sh_q[j] = m.q[gid];
        sh_len[j] = m.length[gid];
        sh_dx[j] = sdn.x;
        sh_n[j] = sdn.y;
        const bool vertical = m.topology[3 * gid] == 2;
        uint32_t lh = P.side_lohi[h3.x + j];
        if (vertical) lh |= kVertical;
        if (!kThetaOne) {
            const int a = (int)(lh & kSlot), b = (int)((lh >> 16) & kSlot);
            const int ga = a ? cbase + ext[a] : 0, gb = b ? cbase + ext[b] : 0;
            const int lower = vertical ? 0 : 2, higher = vertical ? 1 : 3;
            if (m.open_face[4 * ga + lower] > 0.0f || m.open_face[4 * gb + higher] > 0.0f) lh |= kOpen;
            if (a > n_don) sh_nb[j] = face_qn_of(d, ga, lower, m.q);
            if (b > n_don) sh_nb[j] = face_qn_of(d, gb, higher, m.q);
        }
        if (j < n_owned && r.need_side[gid]) lh |= kShared;
        if (kTwo && r.max_hang > 0) {
            const int index = m.edge_index[gid];
            if (index >= 0) {
                Hanging &e = sh_hg[atomicAdd(&sh_hang, 1)];
                e.j = j;
                for (int s = 0; s < 2; ++s) {
                    e.offset[s] = m.offsets[2 * index + s];
                    e.item[s] = e.offset[s] != 0.0f ? 2 * m.slots[2 * index + s] + (vertical ? 1 : 0) : -1;
                    if (e.item[s] >= 0 && d.hang[e.item[s]].cell < 0) e.item[s] = -1;
                }
                lh |= kHangSide;
            }
        }
        sh_lohi[j] = lh;
    }
    // own cells: thread tid has tile offsets tid + NT * k
    int own_slot[CPT], need[CPT], peak[CPT];   // need: 1 depth, 2 face discharges are exchanged
    float rt[CPT], infil[CPT], fastest[CPT], deepest[CPT];
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        const int o = tid + NT * k, slot = o - r0off + 1;
        own_slot[k] = (o >= T || o < r0off || slot > n_r0) ? -1 : slot;
        rt[k] = infil[k] = fastest[k] = deepest[k] = 0.0f;
        need[k] = 0;
        peak[k] = -1;
        if (own_slot[k] < 0) continue;
        const int g = cbase + o;
        rt[k] = m.rain_time[g]; infil[k] = m.infiltration[g];
        fastest[k] = m.max_speed[g]; deepest[k] = m.max_depth[g];
        need[k] = r.need_cell[g];
    }
    __syncthreads();
    const int n_hang = kTwo ? sh_hang : 0;

    // prepare_step (364-371) for trace slot `slot` (one thread)
    auto choose = [&](int slot, uint32_t *row) {
        Clock k = ck;   // the chain runs in registers
        clock_choose(d.min_dt, &k, sh_ndt, row);
        ck = k;
        if (!k.active) return;
        sh_end[slot][0] = k.step_end[0]; sh_end[slot][1] = k.step_end[1];
        for (int b = 0; b < B; ++b) {
            sh_values[b] = sh_coef[2 * b] + sh_coef[2 * b + 1] * (k.local + k.dt / 2.0f);
            sh_levels[b] = sh_coef[2 * b] + sh_coef[2 * b + 1] * k.end_local;
        }
    };
    if (tid == 0) {
        choose(0, blockIdx.x == 0 ? c->trace : sh_row);
        if (ck.active && sh_ndt < limit0 && blockIdx.x == 0) snapshot_limit(d, sh_ndt, sh_arg, &sh_limit);
    }
    if constexpr (kTwo) {
        for (int k = tid; k < 2 * n_hang; k += NT) {
            Hanging &e = sh_hg[k >> 1];
            const int item = e.item[k & 1];
            e.value[k & 1] = item >= 0 ? hang_gradient(d, m.depth, item >> 1, item & 1) : RC(0);
        }
    }
    __syncthreads();
    if (ck.active && sh_ndt < limit0) limit0 = sh_ndt;

    uint32_t epoch = epoch0;
    const int batch = d.batch_size;
    while (ck.active && sh_slot < batch) {
        const float dt = ck.dt;
        const int slot_now = sh_slot;
        const uint32_t step = epoch + 1;            // the words' tag of this step's results
        u64 *depth_words = r.depth_words + (size_t)(epoch & 1u) * m.e_num;
        u64 *side_words = r.side_words + (size_t)(epoch & 1u) * m.s_num;
        if (tid < kBlocks) sh_mask[tid] = 0u;
        if (tid == 0) { sh_near = 0x7f800000u; sh_best = kCflEmpty; }

        if (!kThetaOne) {
            // the discharges beside every side (118-149): of the cells of rings
            // <= 2 from their sides, of ring 3 as they came with the outer rings
            auto beyond = [&](int j, int slot, int face) -> float {
                if (slot == 0) return 0.0f;
                if (slot > n_don) return sh_nb[j];
                const Faces<kTwo> f = faces_of<kTwo>(sh_faces, slot);
                const int a = f.side(face, 0);
                if (!kTwo) return sh_q[a];
                const int b = f.side(face, kTwo ? 1 : 0);
                if (b == n_sides) return sh_q[a];
                return (0.0f + sh_q[a] * sh_len[a] + sh_q[b] * sh_len[b]) / (0.0f + sh_len[a] + sh_len[b]);
            };
            for (int j = tid; j < n_sides; j += NT) {
                const uint32_t lh = sh_lohi[j];
                const int a = (int)(lh & kSlot), b = (int)((lh >> 16) & kSlot);
                const int lower = (lh & kVertical) ? 0 : 2, higher = (lh & kVertical) ? 1 : 3;
                const float left = beyond(j, a, lower), right = beyond(j, b, higher);
                float lext = 0.0f, rext = 0.0f;
                if (lh & kOpen) {
                    lext = m.open_face[a ? 4 * (cbase + ext[a]) + lower : lower];
                    rext = m.open_face[b ? 4 * (cbase + ext[b]) + higher : higher];
                }
                sh_nb[j] = boundary_neighbor_sum(sh_q[j], left, right, lext, rext);
            }
            __syncthreads();
        }

        // P1: momentum (solver_compact.py:439-486) of every local side, the
        // hanging ones after the others
        for (int i = tid; i < n_sides + n_hang; i += NT) {
            int j = i;
            bool hanging = false;
            float part0 = 0.0f, part1 = 0.0f;
            if (kTwo && i >= n_sides) {
                const Hanging &e = sh_hg[i - n_sides];
                j = e.j;
                hanging = true;
                if (e.item[0] >= 0) { d.gradients[e.item[0]] = e.value[0]; part0 = e.value[0] * e.offset[0]; }
                // x - (-y) is x + y, and x - 0 keeps a zero's sign
                if (e.item[1] >= 0) { d.gradients[e.item[1]] = e.value[1]; part1 = -(e.value[1] * e.offset[1]); }
            }
            const uint32_t lh = sh_lohi[j];
            if (kTwo && !hanging && (lh & kHangSide)) continue;
            const int a = (int)(lh & kSlot), b = (int)((lh >> 16) & kSlot);
            const float zl = sh_z[a], zh = sh_z[b], da = sh_h[a], db = sh_h[b];
            const float hl = zl + da, hr = zh + db;
            const float xwh = maxf(hl, hr) - maxf(maxf(zl, zh), kDh);
            float new_q = 0.0f;
            if (!(xwh < d.min_h)) {
                const float xq = sh_q[j], n = sh_n[j];
                float difference = hr - hl;
                if (kTwo && hanging && da > d.min_h && db > d.min_h) difference = difference - part0 - part1;
                const float xdq = (d.neg_g * difference / sh_dx[j]) * maxf(xwh, 0.0f) * dt;
                float ratio = 0.0f;
                if (xq != 0.0f) ratio = xq / friction_pow_real(maxf(xwh, 0.00001f));
                const float xf = 1.0f + d.g * dt * (n * n) * fabsf(ratio);
                const float nb = kThetaOne ? 0.0f + 0.0f : sh_nb[j];
                new_q = (d.sita * xq + d.half_rest * nb + xdq) / xf;
                new_q *= (a == 0) != (b == 0) ? 0.0f : 1.0f;
            }
            sh_q[j] = new_q;
        }
        __syncthreads();

        // P2: donor factor (491-514) of rings <= 2
        {
            uint32_t limited = 0, min_bits = __float_as_uint(1.0f);
            for (int i = 1 + tid; i <= n_don; i += NT) {
                const Faces<kTwo> f = faces_of<kTwo>(sh_faces, i);
                const int bi = sh_bi[i];
                const int kind = bi >= 0 ? sh_kind[bi] : -1;
                float discharge = 0.0f;
                if (kind == 1) discharge = sh_values[bi] * m.weight[cbase + ext[i]];
                const float rainq = sh_rain[i], area = sh_area[i];
                const float pipe = 0.0f;
                const float positive = (maxf(pipe, 0.0f) + maxf(discharge, 0.0f)) * dt;
                const float available = sh_h[i] * area + positive + rainq * dt * area;
                float outgoing = (maxf(-pipe, 0.0f) + maxf(-discharge, 0.0f)) * dt;
#pragma unroll
                for (int dd = 0; dd < 4; ++dd) {
#pragma unroll
                    for (int k = 0; k < (kTwo ? 2 : 1); ++k) {   // a side of no length adds +0
                        const int ls = f.side(dd, k);
                        float signed_q = sh_q[ls] * sh_len[ls];
                        if (dd == 0 || dd == 2) signed_q = -signed_q;
                        outgoing += maxf(signed_q, 0.0f) * dt;
                    }
                }
                float sc = 1.0f;
                if (outgoing > available && kind != 0) {
                    sc = available / outgoing;
                    if (i <= n_r0) {
                        limited += 1;
                        const uint32_t bits = __float_as_uint(sc);
                        min_bits = bits < min_bits ? bits : min_bits;
                    }
                }
                sh_s[i] = sc;
            }
            if (limited) {
                atomicAdd(&sh_cnt[0], limited);
                atomicMin(&sh_minbits, min_bits);
            }
        }
        __syncthreads();

        // the update's inputs from global memory, on their way during P3
        float in_height[CPT], in_width[CPT], in_f0[CPT], in_fc[CPT], in_k[CPT];
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            in_height[k] = in_width[k] = 1.0f;
            in_f0[k] = in_fc[k] = in_k[k] = 0.0f;
            if (own_slot[k] < 0) continue;
            const int g = cbase + tid + NT * k;
            in_height[k] = m.height[g]; in_width[k] = m.width[g];
            if (raining) { in_f0[k] = m.f0[g]; in_fc[k] = m.fc[g]; in_k[k] = m.k[g]; }
        }
        const int first_r1 = n_r0 + 1 + (NT - 1 - tid);   // ring 1 from the last threads, which may own no cell
        float r1_f0 = 0.0f, r1_fc = 0.0f, r1_k = 0.0f;
        if (first_r1 <= n_r01 && raining) {
            const int g = cbase + ext[first_r1];
            r1_f0 = m.f0[g]; r1_fc = m.fc[g]; r1_k = m.k[g];
        }

        // P3: final discharge (516-522) of the faces of rings <= 1; the owned
        // sides that others stage go out
        {
            uint32_t faces = 0;
            for (int j = tid; j < n_qf; j += NT) {
                const uint32_t lh = sh_lohi[j];
                const float q = sh_q[j];
                const float sc = sh_s[q >= 0.0f ? lh & kSlot : (lh >> 16) & kSlot];
                const float qf = q * sc;
                if (j < n_owned) {
                    if (q != 0.0f && sc < 1.0f) faces += 1;
                    if (lh & kShared) put_word(side_words + sh_gid[j], value_word(qf, step));
                }
                sh_q[j] = qf;
            }
            if (faces) atomicAdd(&sh_cnt[1], faces);
        }
        __syncthreads();

        // P4: sources and depth update (525-610)
        float t_removed[CPT], t_floor[CPT], t_level[CPT][5], t_discharge[CPT];
        int t_bi[CPT], t_kind[CPT];
        uint32_t wet = 0;
        auto update = [&](int slot, int g, float f0, float fc, float kh, float &rain_time, float &capacity, float fl[4], float &rain_depth,
                          float &removed, float &floor_v, float &discharge) -> float {
            const Faces<kTwo> f = faces_of<kTwo>(sh_faces, slot);
            const int bi = sh_bi[slot];
            const int kind = bi >= 0 ? sh_kind[bi] : -1;
            const float sc = sh_s[slot], pq = 0.0f;
            const float pipe = maxf(pq, 0.0f) + minf(pq, 0.0f) * sc;
            discharge = 0.0f;
            if (kind == 1) {
                const float requested = sh_values[bi] * m.weight[g];
                discharge = maxf(requested, 0.0f) + minf(requested, 0.0f) * sc;
            }
            const float ssq = pipe + discharge;
            const float rainq = sh_rain[slot];
            if (rainq > 0.0f) {
                rain_time += dt;
                const float diff = f0 - fc;
                capacity = diff == 0.0f ? fc + 0.0f : fc + diff * exp_real(-kh * rain_time / 3600.0f);
            }
#pragma unroll
            for (int dd = 0; dd < 4; ++dd) {
                float face_flux = 0.0f;
#pragma unroll
                for (int k = 0; k < (kTwo ? 2 : 1); ++k) face_flux += sh_q[f.side(dd, k)] * sh_len[f.side(dd, k)];
                fl[dd] = face_flux;
            }
            const float tq = fl[0] - fl[1] + fl[2] - fl[3] + ssq;
            rain_depth = rainq * dt;
            const float flux = tq * dt;
            const float increment = (flux == 0.0f ? flux : flux / sh_area[slot]) + rain_depth;
            float raw_depth = sh_h[slot] + increment;
            removed = minf(capacity * dt, maxf(raw_depth, 0.0f));
            raw_depth -= removed;
            floor_v = maxf(-raw_depth, 0.0f);
            return kind == 0 ? maxf(sh_levels[bi] - sh_z[slot], 0.0f) : maxf(raw_depth, 0.0f);
        };
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            t_removed[k] = t_floor[k] = t_discharge[k] = 0.0f;
            t_bi[k] = t_kind[k] = -1;
#pragma unroll
            for (int e = 0; e < 5; ++e) t_level[k][e] = 0.0f;
            const int slot = own_slot[k];
            if (slot < 0) continue;
            const int o = tid + NT * k, g = cbase + o;
            const int bi = sh_bi[slot], kind = bi >= 0 ? sh_kind[bi] : -1;
            float fl[4], rain_depth, removed, floor_v, discharge;
            const float depth = update(slot, g, in_f0[k], in_fc[k], in_k[k], rt[k], infil[k], fl, rain_depth, removed,
                                       floor_v, discharge);
            if (need[k] & 1) put_word(depth_words + g, value_word(depth, step));
            const float ea = sh_area[slot], previous = sh_h[slot];
            sh_h[slot] = depth;
            t_bi[k] = bi; t_kind[k] = kind;
            t_removed[k] = removed * ea;
            t_floor[k] = floor_v * ea;
            if (kind == 1) t_discharge[k] = discharge * dt;
            if (kind == 0) {
                const float pipe = 0.0f + 0.0f * sh_s[slot];
                t_level[k][0] = (depth - previous) * ea;
                t_level[k][1] = -(fl[0] - fl[1] + fl[2] - fl[3]) * dt;
                t_level[k][2] = -pipe * dt;
                t_level[k][3] = -rain_depth * ea;
                t_level[k][4] = removed * ea;
            }
            const bool is_wet = depth >= d.min_h;
            fastest[k] = fastest_speed(is_wet, fl[0] + fl[1], fl[2] + fl[3], in_height[k], in_width[k],
                                       maxf(depth, 0.01f), fastest[k]);
            if (depth > deepest[k]) {
                deepest[k] = depth;
                peak[k] = slot_now;
            }
            wet += is_wet ? 1u : 0u;
            if (!kThetaOne && (need[k] & 2)) {
                // the cell's face discharges (118-132) for others' next step
                const Faces<kTwo> f = faces_of<kTwo>(sh_faces, slot);
                u64 *out = r.face_words + 4 * ((size_t)(epoch & 1u) * m.e_num + g);
                for (int dd = 0; dd < 4; ++dd) {
                    const int a = f.side(dd, 0), b = kTwo ? f.side(dd, kTwo ? 1 : 0) : n_sides;
                    put_word(out + dd, value_word(b == n_sides ? sh_q[a] : fl[dd] / (0.0f + sh_len[a] + sh_len[b]), step));
                }
            }
            uint32_t mask = 0;
            if (t_removed[k] != 0.0f) mask |= 1u;
            if (t_floor[k] != 0.0f) mask |= kind == 0 ? 4u : 2u;
            if (kind == 0) {
#pragma unroll
                for (int e = 0; e < 5; ++e)
                    if (t_level[k][e] != 0.0f) mask |= 1u << (4 + 5 * bi + e);
            }
            if (kind == 1 && t_discharge[k] != 0.0f) mask |= 1u << (4 + 5 * B + bi);
            if (mask) atomicOr(&sh_mask[o >> 8], mask);
        }
        if (wet) atomicAdd(&sh_cnt[2], wet);
        for (int i = first_r1; i <= n_r01; i += NT) {
            const int g = cbase + ext[i];
            if (i != first_r1 && raining) { r1_f0 = m.f0[g]; r1_fc = m.fc[g]; r1_k = m.k[g]; }
            float2 s = sh_r1[i - n_r0 - 1];
            float fl[4], rain_depth, removed, floor_v, discharge;
            const float depth = update(i, g, r1_f0, r1_fc, r1_k, s.x, s.y, fl, rain_depth, removed, floor_v, discharge);
            sh_r1[i - n_r0 - 1] = s;
            sh_h[i] = depth;
        }
        __syncthreads();

        // P5: CFL (617-641) of the owned sides on the new depths: approximate
        // values first, exact ones only for the sides that may be the block's
        // least (usually one warp's)
        u64 best = kCflEmpty;
        {
            float low = __uint_as_float(0x7f800000u);
            for (int j = tid; j < n_owned; j += NT) {
                const uint32_t lh = sh_lohi[j];
                const int a = (int)(lh & kSlot), b = (int)((lh >> 16) & kSlot);
                if (a == 0 || b == 0) continue;
                const float h = cfl_face_depth(sh_z[a], sh_h[a], sh_z[b], sh_h[b]);
                low = fminf(low, cfl_near(d.afa * sh_len[j], d.g, sh_q[j], h));
            }
            const uint32_t least = __reduce_min_sync(kAll, __float_as_uint(low));
            if (lane == 0) atomicMin(&sh_near, least);
            __syncthreads();
            const float bound = __uint_as_float(sh_near) * kCflMargin;
            if (low <= bound)
                for (int j = tid; j < n_owned; j += NT) {
                    const uint32_t lh = sh_lohi[j];
                    const int a = (int)(lh & kSlot), b = (int)((lh >> 16) & kSlot);
                    if (a == 0 || b == 0) continue;
                    const float h = cfl_face_depth(sh_z[a], sh_h[a], sh_z[b], sh_h[b]);
                    if (cfl_near(d.afa * sh_len[j], d.g, sh_q[j], h) > bound) continue;
                    const u64 key = ((u64)__float_as_uint(cfl_value(d.afa, d.g, sh_len[j], sh_q[j], h)) << 32) | (unsigned)j;
                    // owned sides ascend in id: the lowest local side is the lowest side
                    if (key < sh_best) atomicMin(&sh_best, key);
                }
            __syncthreads();
        }
        int best_side = 0;
        const u64 phase = ((epoch >> 1) & 1u) ? 0ULL : kPhase;
        u64 *keys = r.keys + (size_t)(epoch & 1u) * n_blocks;
        if (warp == 0) {
            best = sh_best;
            best_side = (int)(best & 0xffffffffu);
            best = best == kCflEmpty ? ~kPhase
                                     : (best & 0x7fffffff00000000ULL) | (unsigned)sh_gid[best_side];
            if (lane == 0) put_word(keys + blockIdx.x, best | phase);
        } else if (tid == 32) {
            uint32_t *row = r.counts + 4 * (turn * NHF_MAX_BATCH + slot_now);
            if (sh_cnt[0]) { atomicAdd(row, sh_cnt[0]); atomicMin(row + 3, sh_minbits); }
            if (sh_cnt[1]) atomicAdd(row + 1, sh_cnt[1]);
            if (sh_cnt[2]) atomicAdd(row + 2, sh_cnt[2]);
            sh_cnt[0] = sh_cnt[1] = sh_cnt[2] = 0u; sh_minbits = __float_as_uint(1.0f);
        }

        // budget partials while the words are under way: the canonical tree of
        // each (256-cell block, term) some cell holds, one per warp
        {
            uint32_t any = 0;
#pragma unroll
            for (int k = 0; k < kBlocks; ++k) any |= sh_mask[k];
            while (any) {
                uint32_t chunk = 0;
                int n = 0;
                for (uint32_t rest = any; rest && n < kStage; rest &= rest - 1, ++n) chunk |= rest & (0u - rest);
                any &= ~chunk;
                int jj = 0;
                for (uint32_t rest = chunk; rest; rest &= rest - 1, ++jj) {
                    const int t = __ffs(rest) - 1;
#pragma unroll
                    for (int k = 0; k < CPT; ++k) {
                        const int o = tid + NT * k;
                        if (o >= T) continue;
                        float v = 0.0f;
                        if (t == 0) v = t_removed[k];
                        else if (t == 1) v = t_kind[k] == 0 ? 0.0f : t_floor[k];
                        else if (t == 2) v = t_kind[k] == 0 ? t_floor[k] : 0.0f;
                        else if (t < 4 + 5 * B) {
                            const int q = (t - 4) % 5;
                            if ((t - 4) / 5 == t_bi[k] && t_kind[k] == 0)
                                v = q == 0 ? t_level[k][0] : q == 1 ? t_level[k][1] : q == 2 ? t_level[k][2]
                                  : q == 3 ? t_level[k][3] : t_level[k][4];
                        } else if (t - 4 - 5 * B == t_bi[k]) v = t_discharge[k];
                        sh_stage[jj * T + o] = v;
                    }
                }
                __syncthreads();
                for (int item = kWarps - 1 - warp; item < kBlocks * n; item += kWarps) {   // from the last warp
                    const int hh = item % kBlocks, kk = item / kBlocks;
                    uint32_t rest = chunk;
                    for (int q = 0; q < kk; ++q) rest &= rest - 1;
                    const int t = __ffs(rest) - 1;
                    if (!((sh_mask[hh] >> t) & 1u)) continue;
                    const float *v = sh_stage + kk * T + hh * 256;
                    double sum = (((double)v[lane] + v[lane + 128]) + ((double)v[lane + 64] + v[lane + 192])) +
                                 (((double)v[lane + 32] + v[lane + 160]) + ((double)v[lane + 96] + v[lane + 224]));
                    for (int stride = 16; stride >= 1; stride >>= 1) sum += __shfl_down_sync(kAll, sum, stride);
                    if (lane == 0) acc_add(sh_acc + 2 * (hh * terms_n + t), sh_acc + 2 * (hh * terms_n + t) + 1, sum);
                }
                if (any) __syncthreads();
            }
        }

        bool lost = false;
        if (warp == 0) {
            if (lane == 0) { ck.now[0] = ck.step_end[0]; ck.now[1] = ck.step_end[1]; }   // commit (clock.py:173-181)
            // every block's key: the CFL minimum
            u64 got[kMaxKeys];
#pragma unroll
            for (int k = 0; k < kMaxKeys; ++k) got[k] = lane + 32 * k < n_blocks ? get_word(keys + lane + 32 * k) : phase | ~kPhase;
            u64 least = ~kPhase;
#pragma unroll
            for (int k = 0; k < kMaxKeys; ++k) {
                for (int spin = 0; (got[k] & kPhase) != phase && spin < r.spin_limit && !lost; ++spin)
                    got[k] = get_word(keys + lane + 32 * k);
                lost = lost || (got[k] & kPhase) != phase;
                got[k] &= ~kPhase;
                least = got[k] < least ? got[k] : least;
            }
            least = warp_min_key(least);
            asm volatile("bar.arrive 1, %0;" ::"n"(NT) : "memory");   // the others may look for their words
            const float ndt = least == ~kPhase ? __uint_as_float(0x7f800000u) : __uint_as_float((uint32_t)(least >> 32));
            const int arg = least == ~kPhase ? 0 : (int)(least & 0xffffffffu);
            if (lane == 0) {
                // prepare the batch's next step
                if (blockIdx.x == 0) {
                    uint32_t *row = c->trace + slot_now * NHF_TRACE_COLS;
                    row[0] = __float_as_uint(ck.dt);
                    row[1] = ck.step_end[0]; row[2] = ck.step_end[1];
                    row[3] = NHF_STEP_COMPLETED;
                }
                sh_ndt = ndt; sh_arg = arg;
                if (slot_now + 1 < batch)
                    choose(slot_now + 1, blockIdx.x == 0 ? c->trace + (slot_now + 1) * NHF_TRACE_COLS : sh_row);
                sh_slot = slot_now + 1;
            }
            __syncwarp();
            if (slot_now + 1 < batch && ck.active && ndt < limit0) {
                // the limiting side's snapshot (372-382), by its owner
                limit0 = ndt;
                if (lane == 0) {
                    sh_limit.mine = least == best && least != ~kPhase;
                    if (sh_limit.mine) {
                        const uint32_t lh = sh_lohi[best_side];
                        const int a = (int)(lh & kSlot), b = (int)((lh >> 16) & kSlot);
                        const float h = cfl_face_depth(sh_z[a], sh_h[a], sh_z[b], sh_h[b]);
                        sh_limit.value[0] = ndt;
                        sh_limit.value[1] = sh_h[a]; sh_limit.value[2] = sh_h[b];
                        sh_limit.value[3] = h;
                        sh_limit.value[4] = sh_q[best_side] / rmax(h, RC(1e-30));
                        sh_limit.id[0] = arg; sh_limit.id[1] = cbase + ext[a]; sh_limit.id[2] = cbase + ext[b];
                    }
                }
            }
        } else {
            // the outer rings' new state: depth of rings 2 and 3, discharge of
            // the faces beyond ring 1. With every block's key here the words
            // are (almost always) here too: thousands of warps that poll while
            // they travel would slow them down.
            const int cells = n_ext - 1 - n_r01, all = cells + n_sides - n_qf;
            constexpr int kAhead = 2, kStride = NT - 32;
            const u64 *p[kAhead];
            float *to[kAhead];
            auto addresses = [&](int i) {
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    const int at_k = i + k * kStride, e = n_r01 + 1 + at_k, j = n_qf + at_k - cells;
                    to[k] = at_k >= all ? nullptr : at_k < cells ? sh_h + e : sh_q + j;
                    if (to[k]) p[k] = at_k < cells ? depth_words + cbase + ext[e] : side_words + sbase + srel[j];
                }
            };
            addresses(tid - 32);   // the table reads are over before the keys are here
            asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
            for (int i = tid - 32; i < all; i += kAhead * kStride) {
                u64 w[kAhead];
                if (i != tid - 32) addresses(i);
#pragma unroll
                for (int k = 0; k < kAhead; ++k)
                    if (to[k]) w[k] = get_word(p[k]);
#pragma unroll
                for (int k = 0; k < kAhead; ++k)
                    if (to[k]) *to[k] = await_value(p[k], w[k], step, r.spin_limit, lost);
            }
            if (!kThetaOne) {   // a face of ring 2 towards ring 3: the discharge beyond it
                const u64 *face_words = r.face_words + 4 * (size_t)(epoch & 1u) * m.e_num;
                for (int j = n_qf + tid - 32; j < n_sides; j += kStride) {
                    const uint32_t lh = sh_lohi[j];
                    const int a = (int)(lh & kSlot), b = (int)((lh >> 16) & kSlot);
                    const bool vertical = (lh & kVertical) != 0;
                    if (a <= n_don && b <= n_don) continue;
                    const u64 *p = face_words + (a > n_don ? 4 * (size_t)(cbase + ext[a]) + (vertical ? 0 : 2)
                                                           : 4 * (size_t)(cbase + ext[b]) + (vertical ? 1 : 3));
                    sh_nb[j] = await_value(p, get_word(p), step, r.spin_limit, lost);
                }
            }
            if constexpr (kTwo) {
                for (int k = tid - 32; k < 2 * n_hang; k += kStride) {
                    Hanging &e = sh_hg[k >> 1];
                    const int item = e.item[k & 1];
                    if (item < 0) continue;
                    const HangItem it = d.hang[item];
                    const u64 *p[5];
                    u64 w[5];
                    float h[5], z[5];
                    p[0] = depth_words + it.cell;
#pragma unroll
                    for (int o = 0; o < 4; ++o) p[1 + o] = depth_words + (it.other[o >> 1][o & 1] < 0 ? it.cell : it.other[o >> 1][o & 1]);
#pragma unroll
                    for (int o = 0; o < 5; ++o) { w[o] = get_word(p[o]); z[o] = m.bed[p[o] - depth_words]; }
#pragma unroll
                    for (int o = 0; o < 5; ++o) h[o] = await_value(p[o], w[o], step, r.spin_limit, lost);
                    const real ha[2][2] = {{h[1], h[2]}, {h[3], h[4]}}, za[2][2] = {{z[1], z[2]}, {z[3], z[4]}};
                    e.value[k & 1] = hang_from(it, h[0], z[0], ha, za, d.min_h);
                }
            }
        }
        epoch += 1;
        if (__syncthreads_or(lost)) {   // the batch is void: the host refuses its trace
            if (tid == 0) c->stalled = 1;
            return;
        }
    }

    // ---- the batch's end: state, extrema and budget into the caller's arrays
    for (int i = tid; i < kBlocks * terms_n; i += NT) {
        const int blk = (cbase >> 8) + i / terms_n;
        const size_t g = (size_t)blk * terms_n + i % terms_n;
        if (blk < d.blocks) { d.acc_sum[g] = sh_acc[2 * i]; d.acc_comp[g] = sh_acc[2 * i + 1]; }
    }
    if (tid < 5 && sh_limit.mine) c->limit_value[tid] = sh_limit.value[tid];
    if (tid < 3 && sh_limit.mine) c->limit_ids[tid] = sh_limit.id[tid];
    if (epoch != epoch0)
        for (int j = tid; j < n_owned; j += NT) m.q[sh_gid[j]] = sh_q[j];
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        const int slot = own_slot[k];
        if (slot < 0) continue;
        const int g = cbase + tid + NT * k;
        const float depth = sh_h[slot];
        if (epoch != epoch0) m.depth[g] = depth;
        m.rain_time[g] = rt[k]; m.infiltration[g] = infil[k];
        m.max_speed[g] = fastest[k]; m.max_depth[g] = deepest[k];
        if (peak[k] >= 0) { m.peak_hi[g] = sh_end[peak[k]][0]; m.peak_lo[g] = sh_end[peak[k]][1]; }
        // u, v (solver_compact.py:355-362)
        const Faces<kTwo> f = faces_of<kTwo>(sh_faces, slot);
        float fl[4];
        for (int dd = 0; dd < 4; ++dd) {
            float total = 0.0f;
            for (int e = 0; e < (kTwo ? 2 : 1); ++e) total += sh_q[f.side(dd, e)] * sh_len[f.side(dd, e)];
            fl[dd] = total;
        }
        const float h = maxf(depth, 0.01f);
        float u = 0.0f, v = 0.0f;
        if (depth >= d.min_h) {
            u = (fl[0] + fl[1]) / m.height[g] / h / 2.0f;
            v = (fl[2] + fl[3]) / m.width[g] / h / 2.0f;
        }
        m.u[g] = u; m.v[g] = v;
    }
    // the last block to finish: the steps' counters into the trace and the
    // control block as the step-by-step form leaves it
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        sh_last = atomicAdd(&c->done_blocks, 1u) == (unsigned)n_blocks - 1u;
    }
    __syncthreads();
    if (!sh_last) return;
    __threadfence();
    for (int s = tid; s < NHF_MAX_BATCH; s += NT) {
        if (s < sh_slot) {
            uint32_t *row = c->trace + s * NHF_TRACE_COLS;
            const uint32_t *n = r.counts + 4 * (turn * NHF_MAX_BATCH + s);
            row[6] = __ldcg(n); row[7] = __ldcg(n + 1); row[8] = __ldcg(n + 3); row[9] = __ldcg(n + 2);
        }
        uint32_t *next = r.counts + 4 * ((turn ^ 1u) * NHF_MAX_BATCH + s);
        next[0] = next[1] = next[2] = 0u; next[3] = __float_as_uint(1.0f);
    }
    __syncthreads();
    if (tid == 0) {
        // a clock that stopped says so in every later row
        for (int s = sh_slot + 1; s < batch; ++s) choose(s, c->trace + s * NHF_TRACE_COLS);
        c->now[0] = ck.now[0]; c->now[1] = ck.now[1];
        c->next[0] = ck.next[0]; c->next[1] = ck.next[1];
        c->origin[0] = ck.origin[0]; c->origin[1] = ck.origin[1];
        c->step_end[0] = ck.step_end[0]; c->step_end[1] = ck.step_end[1];
        c->dt = ck.dt; c->local = ck.local; c->end_local = ck.end_local;
        c->active = ck.active; c->slot = batch;
        c->ndt = sh_ndt; c->cfl_arg = sh_arg;
        c->epoch = epoch;
        if (epoch != epoch0) c->grad_parity = 0;
        c->batches += 1;
        c->done_blocks = 0;
    }
}

// Once per solve: which cells' depths (1) and face discharges (2, theta < 1)
// and which sides' discharges some other tile stages, a block per tile; the
// counters' start values.
__global__ void k_resident_setup(const __grid_constant__ Dev d, const __grid_constant__ ResidentArgs r)
{
    const nhf_mesh &m = d.m;
    const int4 *head = r.plan.tile_head + 4 * blockIdx.x;
    const int4 h0 = head[0], h1 = head[1], h2 = head[2], h3 = head[3];
    const int32_t *ext = r.plan.ext_rel + h2.w, *srel = r.plan.side_rel + h3.x;
    for (int i = h0.z + 1 + threadIdx.x; i < h0.x; i += blockDim.x)
        atomicOr(r.need_cell + h2.y + ext[i], !d.theta_one && i > h0.w ? 3 : 1);
    for (int j = threadIdx.x; j < h1.x; j += blockDim.x) {
        const int gid = h2.z + srel[j];
        if (j >= h1.z) r.need_side[gid] = 1;
        const int index = m.hang_cells > 0 ? m.edge_index[gid] : -1;
        if (index < 0) continue;
        for (int s = 0; s < 2; ++s) {
            if (m.offsets[2 * index + s] == 0.0f) continue;
            const HangItem it = d.hang[2 * m.slots[2 * index + s] + (m.topology[3 * gid] == 2 ? 1 : 0)];
            if (it.cell < 0) continue;
            atomicOr(r.need_cell + it.cell, 1);
            for (int o = 0; o < 4; ++o)
                if (it.other[o >> 1][o & 1] >= 0) atomicOr(r.need_cell + it.other[o >> 1][o & 1], 1);
        }
    }
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < 8 * NHF_MAX_BATCH; i += blockDim.x)
            r.counts[i] = (i & 3) == 3 ? __float_as_uint(1.0f) : 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // the words are zero again
        Ctl *c = d.ctl;
        c->epoch = c->batches = 0u;
        c->done_blocks = 0u;
        c->stalled = 0;
    }
}

template <int NT, int T>
void *kernel_of(bool theta_one, bool two)
{
    if (theta_one) return two ? (void *)k_resident<true, true, NT, T> : (void *)k_resident<true, false, NT, T>;
    return two ? (void *)k_resident<false, true, NT, T> : (void *)k_resident<false, false, NT, T>;
}

struct Shape { int threads, tile, stage; void *(*kernel)(bool, bool); };

// The smallest tile that leaves at most one block per SM. More blocks than
// SMs cost more in the exchange than their smaller tiles save (256 x 256
// cells, device time of 32 steps: 129 tiles of 512 cells 343 us, 257 tiles of
// 256 cells, two per SM, 465), and 1024 threads hide latency better than 512
// (83 x 61 cells 233 against 253 us).
const Shape kShapes[] = {
    {1024, 256, 2, kernel_of<1024, 256>},
    {1024, 512, 2, kernel_of<1024, 512>},
    {1024, 768, 1, kernel_of<1024, 768>},
    {1024, 1024, 1, kernel_of<1024, 1024>},
    {1024, 1536, 1, kernel_of<1024, 1536>},
    {1024, 2048, 1, kernel_of<1024, 2048>},
};

}  // namespace

int resident_build(const nhf_mesh &m, int terms, bool theta_one, cudaStream_t s, ResidentBuild *out, char *why,
                   size_t why_len)
{
    auto no = [&](const char *msg) { snprintf(why, why_len, "%s", msg); return 1; };
    if (m.b_num > kMaxBoundaries) return no("more than four boundaries");
    int dev = 0, sms = 0, coop = 0, shared = 0;
    if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) ||
        cudaDeviceGetAttribute(&shared, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) {
        cudaGetLastError();
        return no("device attributes");
    }
    if (!coop) return no("no cooperative launch");
    for (const Shape &shape : kShapes) {
        const int tiles = (m.e_num + shape.tile - 1) / shape.tile;
        if (tiles > sms || tiles > 32 * kMaxKeys) continue;
        TiledBuild tb;
        ResidentArgs r{};
        if (tiled_build(m, s, &tb, why, why_len, shape.tile, 1, &r)) return 1;
        r.plan = tb.plan;
        if (r.max_per_face > 2) { cudaFree(tb.device_memory); return no("a face of more than two sides"); }
        const bool two = r.max_per_face > 1 || m.hang_cells > 0;
        void *kernel = shape.kernel(theta_one, two);
        const size_t smem = sizes_of(r, terms, theta_one, two ? 2 : 1, shape.stage).total;
        int per_sm = 0;
        cudaFuncAttributes fa;
        if (r.plan.max_ext > (int)kSlot || cudaFuncGetAttributes(&fa, kernel) != cudaSuccess ||
            smem + fa.sharedSizeBytes > (size_t)shared ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shared - (int)fa.sharedSizeBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, shape.threads, smem) != cudaSuccess ||
            (long long)per_sm * sms < tiles) {
            // a larger tile needs more shared memory still
            cudaGetLastError();
            cudaFree(tb.device_memory);
            return no("tiles do not fit the GPU at once");
        }
        // two buffers of words (keys, depths, sides, for theta < 1 face
        // discharges), two of counters, the exchange flags
        size_t off = 0;
        auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 255) & ~size_t(255); return o; };
        const size_t e = m.e_num, sn = m.s_num;
        const size_t o_key = take(16 * (size_t)tiles), o_dep = take(16 * e), o_side = take(16 * sn);
        const size_t o_face = take(theta_one ? 0 : 64 * e), o_cnt = take(32 * NHF_MAX_BATCH);
        const size_t o_nc = take(4 * e), o_ns = take(sn);
        char *mem = nullptr;
        if (cudaMalloc((void **)&mem, off) || cudaMemsetAsync(mem, 0, off, s)) {
            cudaGetLastError();
            if (mem) cudaFree(mem);
            cudaFree(tb.device_memory);
            return no("no device memory for the resident form");
        }
        r.spin_limit = kSpinLimit;
        r.keys = (unsigned long long *)(mem + o_key);
        r.depth_words = (unsigned long long *)(mem + o_dep);
        r.side_words = (unsigned long long *)(mem + o_side);
        r.face_words = (unsigned long long *)(mem + o_face);
        r.counts = (uint32_t *)(mem + o_cnt);
        r.need_cell = (int32_t *)(mem + o_nc);
        r.need_side = (uint8_t *)(mem + o_ns);
        out->args = r;
        out->words_bytes = o_cnt;
        out->tables = tb.device_memory;
        out->memory = mem;
        out->kernel = kernel;
        out->threads = shape.threads;
        out->shared_bytes = smem;
        out->patterns = tb.patterns;
        return 0;
    }
    return no("tiles do not fit the GPU at once");
}

cudaError_t resident_enqueue_setup(const Dev &d, ResidentBuild &b, cudaStream_t s)
{
    const char *spins = getenv("NHF_RESIDENT_SPINS");
    b.args.spin_limit = spins && atoi(spins) >= 0 ? atoi(spins) : kSpinLimit;
    const cudaError_t e = cudaMemsetAsync(b.memory, 0, b.words_bytes, s);
    if (e != cudaSuccess) return e;
    k_resident_setup<<<b.args.plan.n_tiles, 256, 0, s>>>(d, b.args);
    return cudaGetLastError();
}

cudaError_t resident_enqueue_batch(const Dev &d, const ResidentBuild &b, const uint32_t words[4], cudaStream_t s)
{
    ResidentArgs r = b.args;
    for (int k = 0; k < 4; ++k) r.words[k] = words[k];
    Dev dev = d;
    void *args[2] = {&dev, &r};
    return cudaLaunchCooperativeKernel(b.kernel, dim3(r.plan.n_tiles), dim3(b.threads), args, b.shared_bytes, s);
}

}  // namespace nhf

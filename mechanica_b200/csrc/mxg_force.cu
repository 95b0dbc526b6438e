/*
 * Nonbonded forces by columns: the force pass of spaces whose cells are cubic and at least the
 * cutoff wide (the 27-cell neighbourhood, each pair of cells once in the reference's task list).
 *
 * Cells that share x and y are consecutive in the slot order, so a column's particles are one run
 * of slots, and so are three neighbouring cells along z. A warp takes up to 32 consecutive
 * particles of a column, one per lane, and sums each one's force over all its neighbours: every
 * pair is evaluated once from each side (the two evaluations are exact negations), so a force is
 * complete when the lane's sum is, with no received sums to store, add up later or order.
 *
 *   1. Staging. The particles of the nine columns around within a cell of the warp's z range are
 *      loaded (runs of consecutive slots), those beyond the cutoff of the bounding box of the
 *      warp's own particles are dropped, the rest are compacted into shared memory.
 *   2. Candidates. 32 staged particles at a time sit one per lane in registers, the own particles
 *      come one after another from shared memory; a ballot gives the own particle's lane 32 bits
 *      of its neighbours. The squared distance is |a|^2 + |b|^2 - 2 a.b, three fused multiply-adds,
 *      against a cutoff widened by more than its rounding: a superset, the exact test follows.
 *   3. Pairs. Each lane walks its own bits, reads the neighbour from shared memory and adds the
 *      pair's force to its registers. All nine columns are walked together: the number of neighbours
 *      in a part of the sphere varies far more from lane to lane than their total.
 *
 * Positions are staged as integers, units of a power of two near 2^-27 of a cell edge from the
 * middle of the warp's cells: cell-relative FP32 positions convert exactly down to that unit, the
 * shift of a neighbour cell is an addition without rounding, and a pair's displacement is the same
 * from both sides, up to its sign, to the bit. The arithmetic below is in these units. 32 bits hold
 * the kColumnSpan cells that a warp's particles may span and those on both sides of them: longer
 * columns are cut into parts of that length, so the unit is the same for every warp of a space.
 *
 * The sums' order is fixed by the column's own content and the number of warps that share a group,
 * so results do not depend on scheduling. That number follows the engine's particles (or a pinned
 * variant), and the instantiation and the choice of this kernel what potentials the engine has: with
 * all of them alike, a replica has the bits that it has alone.
 *
 * Bound: instruction issue and latency. A DPD pass over 200,000 particles in 16,000 cells of the cutoff: 129 us,
 * 74.4 M warp instructions, 57 % of the issue slots, 14 warps a SM (16 by the staged particles' shared memory); by
 * leaving phases out, setting up and staging 49 us, candidates 34, pairs 50.
 * Force pass with the cell kernel (mxg_kernels.cu) / this one: Lennard-Jones, 270,000 particles in cells of
 * 1.0 / 1.67 / 2.5 cutoffs: 204 / 511 / 1,163 -> 154 / 231 / 418 us; 10,000 in the default 4^3 cells: 208 -> 39;
 * DPD, density 3, 192,000: 172 -> 72; density 13, 832,000: 585 -> 462, and 30 us less in the integrator, which has no
 * received sums to add. Chains, 20,360: 40 -> 34; 3,375 DPD particles: 23 -> 15.
 */
#include <algorithm>

#include "mxg_device.cuh"
#include "mxg_kernels.h"

namespace mxg {

namespace {

constexpr unsigned kFull = 0xffffffffu;

/* What the force terms of an engine can be: tables only; tables, DPD, summed second terms, Philox;
 * DPD only with the reference's random term. */
enum : int { kTerms = 0, kTermsDpd = 1, kTermsPureDpd = 2, kTermsFlux = 3 };  // the last: species fluxes, no forces
__host__ __device__ constexpr bool needs_velocities(int kind) { return kind == kTermsDpd || kind == kTermsPureDpd; }

template <int kKind>
struct ColSmem {
    static constexpr int kCap = needs_velocities(kKind) ? 288 : 448;          // staged particles (a multiple of 32)
    int4 nb[kCap + 1];                               // staged position; w = (z + 1) << 11 | code << 6 | type
    float4 nb_v[needs_velocities(kKind) ? kCap + 1 : 1];  // velocity, w = id
    ulonglong2 own_xy[32], own_zr[32];           // candidate test: pairs of -2 x, -2 y, -2 z; widened cutoff^2 - |x|^2
    unsigned mask[kCap / 32 + 1][32];            // neighbours found, per group of 32 staged and own particle
    int4 run[27];                                // runs of slots staged: first slot less offset, end, cell base, code
    int4 off[27];                                // and their shift from the warp's frame, in units
    int slot[kKind == kTermsPureDpd ? 1 : kCap]; // slot of the staged particle (for odd_pairs); fluxes: its id
    float rate[kKind == kTermsFlux ? 8 : 1][32];  // fluxes: the own particles' rates
    int self[32];                                // own particle's staged index in this region, or -1
};

/* A type pair's potential, as EngineView::pair_rec describes it. */
struct PairRec {
    float4 p, q;
    __device__ __forceinline__ int code() const { return __float_as_int(q.w); }
};
__device__ __forceinline__ PairRec load_rec(const float4 *rec, int pk) {
    PairRec r;
    r.p = __ldg(rec + 3 * pk);
    r.q = __ldg(rec + 3 * pk + 1);
    return r;
}

/* 1 / sqrt without the handling of denormals. */
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* Potential and force of a table at r2 >= a^2 and not past its end (potential_eval_ex, potential_eval.hpp:
 * 106-161; e and f = V'(r) / r): false out of range. Fused multiply-adds, and the square root and the
 * division by r from one reciprocal square root with a Newton step for r. */
__device__ __forceinline__ bool table_term(const PairRec &rec, const float *__restrict__ coef, float r2, float &e, float &f) {
    const float r2c = fmaxf(r2, 1.42108547e-14f);  // the reference's lower bound on r, FLT_EPSILON
    const float ir = rsqrt_ftz(r2c);
    float r = __fmul_rn(r2c, ir);
    r = __fmaf_rn(__fmaf_rn(-r, r, r2c), 0.5f * ir, r);
    const float s = __fmaf_rn(r, rec.p.y, rec.p.z);
    const float t = __fmaf_rn(s, __fmaf_rn(s, rec.q.z, rec.q.y), rec.q.x);
    const unsigned ind = (unsigned)fmaxf(0.0f, t);
    const unsigned code = (unsigned)max(rec.code(), 0), count = code >> 20;
    const bool in = ind <= count;  // no branch: the last interval's values are not used
    const float4 *c4 = reinterpret_cast<const float4 *>(coef) + 2 * ((code & 0xfffffu) + min(ind, count));
    const float4 c0 = __ldg(c4), c1 = __ldg(c4 + 1);
    const float x = __fmul_rn(__fsub_rn(s, c0.x), c0.y);
    float ee = __fmaf_rn(c0.z, x, c0.w), eff = c0.z;
    eff = __fmaf_rn(eff, x, ee); ee = __fmaf_rn(ee, x, c1.x);
    eff = __fmaf_rn(eff, x, ee); ee = __fmaf_rn(ee, x, c1.y);
    eff = __fmaf_rn(eff, x, ee); ee = __fmaf_rn(ee, x, c1.z);
    eff = __fmaf_rn(eff, x, ee); ee = __fmaf_rn(ee, x, c1.w);
    e = ee;
    f = __fmul_rn(__fmul_rn(eff, c0.y), ir);
    return in;
}

/* dpd_eval (dpd_eval.hpp:21-69) as f / r, for the force f d / r on the particle d points to:
 * oc (alpha + sigma delta xi - gamma oc (e.v)), oc = 1 - r/rc, e = d/r, v the relative velocity. */
__device__ __forceinline__ float dpd_term(float oc, float ir, float dv, float gamma, float drive) {
    return __fmul_rn(__fmul_rn(oc, __fmaf_rn(__fmul_rn(-gamma, oc), __fmul_rn(dv, ir), drive)), ir);
}

/* The DPD term of a pair (rec its potential, d from the neighbour to the own particle): the own
 * particle's force is fs * d. False out of range. */
__device__ __forceinline__ bool pair_dpd(const EngineView &v, const PairRec &rec, float dx, float dy, float dz, float r2,
                                         const float4 &vi, const float4 &vj, unsigned rng_mode, float &fs) {
    if (r2 > __fmul_rn(rec.p.y, rec.p.y) || rec.code() == -2) return false;
    // r, 1/r and the quotient by the cutoff one Newton step on from the unit's results: as close to
    // the FP64 values as divisions (DPD mixed with tables, shifted, or with the Philox stream)
    float ir = rsqrt_ftz(r2);
    float r = __fmul_rn(r2, ir);
    r = __fmaf_rn(__fmaf_rn(-r, r, r2), 0.5f * ir, r);
    ir = __fmaf_rn(__fmaf_rn(-r, ir, 1.0f), ir, ir);
    const float sr = __fsub_rn(r, rec.p.w), qt = __fmul_rn(sr, rec.p.z);
    const float oc = sr < 0.f ? 1.f : __fmaf_rn(__fmaf_rn(qt, rec.p.y, -sr), rec.p.z, __fsub_rn(1.0f, qt));
    const float dv = __fmaf_rn(dx, __fsub_rn(vi.x, vj.x),
                               __fmaf_rn(dy, __fsub_rn(vi.y, vj.y), __fmul_rn(dz, __fsub_rn(vi.z, vj.z))));
    float xi = 1.f;
    if (rng_mode) {
        const unsigned idi = __float_as_uint(vi.w), idj = __float_as_uint(vj.w);
        xi = philox_pair_xi(*v.step, min(idi, idj), max(idi, idj));
    }
    fs = dpd_term(oc, ir, dv, rec.q.y, __fmaf_rn(rec.q.z, xi, rec.q.x));
    return true;
}

/* One term of a pair in an engine of tables and DPD: the own particle's force is fs * d. False out of
 * range; edge: so near to a table's end that rounding decides on which side of it the pair is. */
__device__ __forceinline__ bool pair_term(const EngineView &v, const PairRec &rec, float dx, float dy, float dz, float r2,
                                          const float4 &vi, const float4 &vj, unsigned rng_mode, float &fs, float &e,
                                          bool &edge) {
    e = 0.f;
    edge = false;
    if (rec.code() < 0) return pair_dpd(v, rec, dx, dy, dz, r2, vi, vj, rng_mode, fs);
    const bool in = table_term(rec, v.coef, r2, e, fs);
    fs = -fs;
    edge = r2 > rec.p.w && r2 <= rec.p.w * v.near_ratio;
    return in && r2 <= rec.p.w;
}

/* potential_eval_ex in its own arithmetic, for the pairs of odd_pairs; x: the record's third part. It is
 * loaded with the others: the chain of loads of one such pair is as long as the kernel's last warp. */
__device__ __forceinline__ bool table_reference(const PairRec &rec, const float4 &x, const float *__restrict__ coef, float r2,
                                                float &e, float &f) {
    const float r = __fsqrt_rn(r2), ro = fmaxf(r, 1.19209290e-7f), ra = fmaxf(r, __fsqrt_rn(x.x));
    const float s = x.w < 0.f ? __fdiv_rn(ra, -x.w) : __fadd_rn(__fsub_rn(ra, x.w), x.z);
    const float t = __fadd_rn(rec.q.x, __fmul_rn(s, __fadd_rn(rec.q.y, __fmul_rn(s, rec.q.z))));
    const unsigned ind = (unsigned)fmaxf(0.0f, t), code = (unsigned)rec.code();
    if (s > x.y || ind > code >> 20) return false;
    const float4 *c4 = reinterpret_cast<const float4 *>(coef) + 2 * ((code & 0xfffffu) + ind);
    const float4 c0 = __ldg(c4), c1 = __ldg(c4 + 1);
    const float u = __fmul_rn(__fsub_rn(s, c0.x), c0.y);
    float ee = __fadd_rn(__fmul_rn(c0.z, u), c0.w), eff = c0.z;
    eff = __fadd_rn(__fmul_rn(eff, u), ee); ee = __fadd_rn(__fmul_rn(ee, u), c1.x);
    eff = __fadd_rn(__fmul_rn(eff, u), ee); ee = __fadd_rn(__fmul_rn(ee, u), c1.y);
    eff = __fadd_rn(__fmul_rn(eff, u), ee); ee = __fadd_rn(__fmul_rn(ee, u), c1.z);
    eff = __fadd_rn(__fmul_rn(eff, u), ee); ee = __fadd_rn(__fmul_rn(ee, u), c1.w);
    e = ee;
    f = __fdiv_rn(__fmul_rn(eff, c0.y), ro);
    return true;
}

/* pair_term for the pairs of odd_pairs. */
template <int kKind>
__device__ __forceinline__ bool odd_term(const EngineView &v, const PairRec &rec, const float4 &x, const float3 &d, float r2,
                                         const float4 &vi, const float4 &vj, unsigned rng_mode, float &fs, float &e) {
    e = 0.f;
    if (kKind != kTerms && rec.code() < 0) return pair_dpd(v, rec, d.x, d.y, d.z, r2, vi, vj, rng_mode, fs);
    if (kKind == kTermsPureDpd || !table_reference(rec, x, v.coef, r2, e, fs)) return false;
    fs = -fs;
    return true;
}

/* A random direction of length a for a pair closer than a (potential_eval_super_ex, dpd_eval.hpp:
 * 122-131), here a Philox draw keyed on the step and the two ids. */
__device__ __forceinline__ float3 close_pair(const EngineView &v, unsigned idi, unsigned idj, float a) {
    float g0, g1, g2;
    philox_normal3(*v.step, min(idi, idj), max(idi, idj), g0, g1, g2);
    const float k = (idi < idj ? a : -a) / sqrtf(g0 * g0 + g1 * g1 + g2 * g2);
    return make_float3(g0 * k, g1 * k, g2 * k);
}

/* The cell at offset (ox, oy, oz) from the cell at (x, y, z) of the replica and the shift between
 * them; -1 where the box ends. */
__device__ __forceinline__ int neighbour_cell(const DevSpace &S, int x, int y, int z, int ox, int oy, int oz, float s[3]) {
    int l[3] = {x + ox, y + oy, z + oz};
    const int o[3] = {ox, oy, oz};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s[k] = (float)o[k] * S.sh[k];
        if (l[k] < 0 || l[k] >= S.cdim[k]) {
            if (!((S.periodic >> k) & 1)) return -1;
            l[k] += l[k] < 0 ? S.cdim[k] : -S.cdim[k];
            s[k] = (float)o[k] * S.shw[k];
        }
    }
    return S.cell_offset + (l[0] * S.cdim[1] + l[1]) * S.cdim[2] + l[2];
}

/* The reference skips a pair of cells as a whole when the largest projection key of its first cell,
 * along the pair's sort direction, exceeds the smallest of its second plus the shift's
 * (runner_dopair.cpp:167-171, an unsigned difference that wraps): particles within a key quantum of
 * a shared face, edge or corner, or outside their cell. (The test's other side, cells further apart
 * than the cutoff, never drops a pair inside the cutoff of cubic cells.) */
__device__ __noinline__ bool cells_skipped(const EngineView &v, const DevSpace &S, int x, int y, int z, int ox, int oy,
                                           int oz) {
    const int code = (ox + 1) * 9 + (oy + 1) * 3 + (oz + 1);
    if (code == 13) return false;
    float s[3];
    const int c = S.cell_offset + (x * S.cdim[1] + y) * S.cdim[2] + z;
    const int nc = neighbour_cell(S, x, y, z, ox, oy, oz, s);
    if (nc < 0 || v.cell_count[nc] == 0 || v.cell_count[c] == 0) return false;
    // the pair's first cell is the one whose offset to the other is positive (space_getsid's flip);
    // the sort directions are numbered by the negative offsets
    const int sid = code < 13 ? code : 26 - code;
    const int first = code < 13 ? nc : c, second = code < 13 ? c : nc;
    const int dn = (int)__fmul_rn(S.sort_dscale, __fsqrt_rn(dot3_rn(s[0], s[1], s[2])));
    return v.sort_bounds[second * 13 + sid].x + dn - v.sort_bounds[first * 13 + sid].y < 0;
}

/* Whether any pair of cells between the warp's cells (column x, y, z0 to z1) that hold particles near a
 * face and their neighbours is skipped. Same result in all lanes. */
__device__ __noinline__ bool any_skipped(const EngineView &v, const DevSpace &S, int x, int y, int z0, int z1) {
    const int lane = threadIdx.x & 31;
    bool skip = false;
    for (int z = z0; z <= z1; ++z) {
        if (!v.cell_near[S.cell_offset + (x * S.cdim[1] + y) * S.cdim[2] + z]) continue;
        if (lane < 27) skip |= cells_skipped(v, S, x, y, z, lane / 9 - 1, lane / 3 % 3 - 1, lane % 3 - 1);
    }
    return __any_sync(kFull, skip);
}

/* For warps whose cells may be part of a skipped pair of cells, or whose particles may lie outside
 * their cells: takes the bits of pairs that the reference's task list does not reach out of the
 * masks. Rare, so a walk of its own. */
template <int kKind>
__device__ __noinline__ void drop_unreached(const EngineView &v, ColSmem<kKind> &sm, const DevSpace &S, int x, int y, int z,
                                            int zrel, int ngroups, bool live) {
    const int lane = threadIdx.x & 31;
    for (int u = 0; u < ngroups; ++u) {
        unsigned bits = live ? sm.mask[u][lane] : 0u, keep = bits;
        while (bits) {
            const int b = __ffs(bits) - 1, w = sm.nb[u * 32 + b].w;
            bits &= bits - 1u;
            const int dz = (w >> 11) - 1 - zrel, code = (w >> 6) & 31;
            if (dz < -1 || dz > 1 ||
                ((S.prune & 2) && cells_skipped(v, S, x, y, z, code % 9 / 3 - 1, code % 3 - 1, dz)))
                keep &= ~(1u << b);
        }
        sm.mask[u][lane] = keep;
    }
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

/* Two FP32 fused multiply-adds in one instruction. */
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(a));
    return d;
}

/* Candidate bits of 2 kU groups of 32 staged particles from group u0 on, for every own particle, into
 * mask (the last group may lie past ngrp: its bits are empty). Bound: instruction issue; a pair of
 * groups takes three packed multiply-adds and, for each, a compare, a ballot and a select. */
template <int kKind, int kU>
__device__ __forceinline__ void candidates(ColSmem<kKind> &sm, int u0, int base, int nown) {
    const int lane = threadIdx.x & 31;
    unsigned long long x[kU], y[kU], z[kU], s[kU];
    unsigned m[2 * kU];
#pragma unroll
    for (int k = 0; k < kU; ++k) {
        float c[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int idx = (u0 + 2 * k + h) * 32 + lane;
            c[h][0] = c[h][1] = c[h][2] = 0.f;
            c[h][3] = __int_as_float(0x7f800000);  // an empty place is never within reach
            m[2 * k + h] = 0u;
            if (idx < base) {
                const int4 q = sm.nb[idx];
                c[h][0] = (float)q.x;
                c[h][1] = (float)q.y;
                c[h][2] = (float)q.z;
                c[h][3] = __fmaf_rn(c[h][0], c[h][0], __fmaf_rn(c[h][1], c[h][1], c[h][2] * c[h][2]));
            }
        }
        x[k] = pack2(c[0][0], c[1][0]);
        y[k] = pack2(c[0][1], c[1][1]);
        z[k] = pack2(c[0][2], c[1][2]);
        s[k] = pack2(c[0][3], c[1][3]);
    }
#pragma unroll 4
    for (int il = 0; il < nown; ++il) {
        const ulonglong2 txy = sm.own_xy[il];  // (-2 x, -2 x), (-2 y, -2 y)
        const ulonglong2 tzr = sm.own_zr[il];  // (-2 z, -2 z), (the cutoff side, 0)
        const float reach = unpack2(tzr.y).x;
#pragma unroll
        for (int k = 0; k < kU; ++k) {
            const float2 d = unpack2(fma2(txy.x, x[k], fma2(txy.y, y[k], fma2(tzr.x, z[k], s[k]))));
            const unsigned b0 = __ballot_sync(kFull, d.x <= reach), b1 = __ballot_sync(kFull, d.y <= reach);
            m[2 * k] = lane == il ? b0 : m[2 * k];
            m[2 * k + 1] = lane == il ? b1 : m[2 * k + 1];
        }
    }
#pragma unroll
    for (int k = 0; k < 2 * kU; ++k) sm.mask[u0 + k][lane] = m[k];
}

/* z in the warp's frame; the sum may pass 2^31 on the way (at most kColumnSpan + 1 edges below 2^27 each). */
__device__ __forceinline__ int column_z(int z, int cells, int edge, int off) {
    return (int)((unsigned)z + (unsigned)cells * (unsigned)edge + (unsigned)off);
}

/* Whether a cell-relative position is finite and near enough to its cell (7 edges, far) for its integer
 * form, which has no other value for the rest; a particle that is not has no neighbours. */
__device__ __forceinline__ bool on_grid(const float4 &x, float far) { return fabsf(x.x) + fabsf(x.y) + fabsf(x.z) <= far; }

/* A lane's sums over the pairs it walks. */
struct ColSums {
    float x, y, z;
    double e;
};

/* What a lane needs of its own particle. */
struct ColOwn {
    int x, y, z, zrel, type, slot;
    float4 vel;
};

/* The displacement from the particle at slot_j to the one at slot_i as the reference rounds it, d =
 * (x_first - s) - x_second from the cell-relative positions; side orders the two cells (0: the same cell,
 * > 0: that of slot_i is the first), c9 and oz are the other cell's place among the nine columns and
 * along z, (x, y, z) the own cell. */
__device__ __forceinline__ float3 reference_d(const EngineView &v, const DevSpace &S, int slot_i, int slot_j, int x, int y,
                                              int z, int c9, int oz, int side) {
    const float4 xi = v.pos[slot_i], xj = v.pos[slot_j];
    float s[3] = {0.f, 0.f, 0.f};
    if (side != 0) neighbour_cell(S, x, y, z, c9 / 3 - 1, c9 % 3 - 1, oz, s);
    return side < 0 ? make_float3(__fsub_rn(xi.x, __fadd_rn(xj.x, s[0])), __fsub_rn(xi.y, __fadd_rn(xj.y, s[1])),
                                  __fsub_rn(xi.z, __fadd_rn(xj.z, s[2])))
                    : make_float3(__fsub_rn(__fsub_rn(xi.x, s[0]), xj.x), __fsub_rn(__fsub_rn(xi.y, s[1]), xj.y),
                                  __fsub_rn(__fsub_rn(xi.z, s[2]), xj.z));
}

/* Whether the reference counts a pair near the cutoff as within it (its cell loop's cutoff for pairs of
 * one cell, its pair loop's for others). */
__device__ __noinline__ bool reference_within(const EngineView &v, const DevSpace &S, int slot_i, int slot_j, int x, int y,
                                              int z, int c9, int oz, int side) {
    const float3 d = reference_d(v, S, slot_i, slot_j, x, y, z, c9, oz, side);
    return dot3_rn(d.x, d.y, d.z) <= (side == 0 ? S.cut2_self : S.cut2_pair);
}

/* The pairs that the main walk leaves out: those closer than their potential's a, which get a random
 * direction of that length, those so near to a, to the cutoff or to a table's end that the decision depends
 * on rounding (in a DPD-only pass the force vanishes at the cutoff, and only a counts), and those closer
 * than kClose2. They take the reference's displacement, r^2 unfused, and its evaluation of a table. The main
 * walk clears a lane's bits as it takes them and sets these again; rare, so a walk of its own. */
template <int kKind>
__device__ __noinline__ ColSums odd_pairs(const EngineView &v, ColSmem<kKind> &sm, const DevSpace &S, ColOwn o, int x, int y,
                                          int z, int ngroups, bool live) {
    const int lane = threadIdx.x & 31;
    ColSums sum = {0.f, 0.f, 0.f, 0.0};
    for (int u = 0; u < ngroups; ++u) {
        unsigned bits = live ? sm.mask[u][lane] : 0u;
        while (bits) {
            const int jj = u * 32 + __ffs(bits) - 1;
            bits &= bits - 1u;
            const int4 b = sm.nb[jj];
            const int pk = S.pot_offset + o.type * v.ntypes + (b.w & 63);
            const PairRec rec = load_rec(v.pair_rec, pk);
            if (rec.code() == -2) continue;
            const float4 x3 = __ldg(v.pair_rec + 3 * pk + 2);
            const int slot_j = kKind == kTermsPureDpd ? v.slot_of_id[__float_as_int(sm.nb_v[jj].w)] : sm.slot[jj];
            const int c9 = ((b.w >> 6) & 31) % 9, oz = (b.w >> 11) - 1 - o.zrel;
            const int side = (c9 / 3 - 1) * 9 + (c9 % 3 - 1) * 3 + oz;  // 0: own cell, > 0: the first of the two
            const float cut2 = side == 0 ? S.cut2_self : S.cut2_pair;
            const float3 d = reference_d(v, S, o.slot, slot_j, x, y, z, c9, oz, side);
            const float r2 = dot3_rn(d.x, d.y, d.z);
            if (r2 > cut2) continue;
            const float4 vj = kKind != kTerms ? sm.nb_v[jj] : make_float4(0.f, 0.f, 0.f, 0.f);
            float3 t = d;
            if (r2 < x3.x) {
                const unsigned idi = __float_as_uint(kKind != kTerms ? o.vel.w : v.vel[o.slot].w);
                const unsigned idj = __float_as_uint(kKind != kTerms ? vj.w : v.vel[sm.slot[jj]].w);
                t = close_pair(v, idi, idj, sqrtf(x3.x));
            }
            float fs = 0.f, e = 0.f;
            if (!odd_term<kKind>(v, rec, x3, t, fmaxf(r2, x3.x), o.vel, vj, S.rng_mode, fs, e)) fs = e = 0.f;
            sum.x += fs * t.x;
            sum.y += fs * t.y;
            sum.z += fs * t.z;
            sum.e += (double)e;
            if (kKind == kTermsDpd && v.pot_idx2) {  // a second potential acts on the pair's own displacement
                const PairRec rec2 = load_rec(v.pair_rec2, pk);
                const float4 y3 = __ldg(v.pair_rec2 + 3 * pk + 2);
                if (rec2.code() != -2 && !(r2 < y3.x) && odd_term<kKind>(v, rec2, y3, d, r2, o.vel, vj, S.rng_mode, fs, e)) {
                    sum.x += fs * d.x;
                    sum.y += fs * d.y;
                    sum.z += fs * d.z;
                    sum.e += (double)e;
                }
            }
        }
    }
    return sum;
}

/* The species fluxes of one pair, seen from the own particle. The kernel's third use: the staging and the
 * candidates find the pairs, the values are gathered by id. Bound: the latency of those gathers. 50,021
 * particles of 4 in a cell, 17 neighbours each, five flux entries over three type pairs: 213 us with one
 * thread a particle walking 27 cells (flux_kernel, kept for other spaces), 66 us here.
 * flux_eval_ex (flux_eval.hpp:33-84): weight
 * (1 - r/cutoff)^2 formed in FP64 from the FP32 distance as there, q from the entry's a to its b particle
 * (the pair's first is a when both types are), decay from both. own_first: in the reference's order. */
template <int kKind>
__device__ __forceinline__ void pair_fluxes(const EngineView &v, const SpeciesView &sp, ColSmem<kKind> &sm, int lane, int id,
                                            int type, int id_j, int type_j, bool own_first, float r, double inv_cutoff) {
    const int t1 = own_first ? type : type_j, t2 = own_first ? type_j : type;
    const int f0 = sp.flux_off[t1 * v.ntypes + t2], f1 = sp.flux_off[t1 * v.ntypes + t2 + 1];
    if (f0 == f1) return;
    float w = (float)__fma_rn(-(double)r, inv_cutoff, 1.0);
    w = __fmul_rn(w, w);
    const int id1 = own_first ? id : id_j, id2 = own_first ? id_j : id;
    for (int q = f0; q < f1; ++q) {
        const DevFlux &F = sp.flux[q];
        const int ida = t1 == F.ta ? id1 : id2, idb = t2 == F.tb ? id2 : id1;
        const float sa = sp.value[(size_t)ida * sp.smax + F.ia], sb = sp.value[(size_t)idb * sp.smax + F.ib];
        float g;
        if (F.kind == 0)
            g = __fmul_rn(F.k, __fsub_rn(sa, sb));
        else {  // times 0 or 1, so that values that are not finite reach both particles
            const float u = F.kind == 1 ? __fmul_rn(F.k, __fsub_rn(sa, F.target))
                                        : __fmul_rn(__fmul_rn(F.k, __fsub_rn(F.target, sb)), sa);
            g = __fmul_rn(u > 0.f ? 1.f : 0.f, u);
        }
        const float qq = __fmul_rn(w, g), hd = __fmul_rn(F.decay, 0.5f);
        if (ida == id) sm.rate[F.ia][lane] = __fsub_rn(__fsub_rn(sm.rate[F.ia][lane], qq), __fmul_rn(hd, sa));
        if (idb == id) sm.rate[F.ib][lane] = __fsub_rn(__fadd_rn(sm.rate[F.ib][lane], qq), __fmul_rn(hd, sb));
    }
}

/* kSplit warps of a block share a group of particles: each takes every kSplit-th 64 of the particles to
 * be staged, and their sums are added in order. */
template <int kKind, int kSplit>
__global__ void __launch_bounds__(32 * kSplit, 18 / kSplit) column_force_kernel(const __grid_constant__ EngineView v,
                                                                              const __grid_constant__ SpeciesView sp) {
    using Smem = ColSmem<kKind>;
    extern __shared__ float4 col_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Smem &sm = reinterpret_cast<Smem *>(col_smem)[w];
    const unsigned lt_mask = (1u << lane) - 1u;
    const int ntypes = v.ntypes;
    for (int it = blockIdx.x; it < v.ncol_items; it += gridDim.x) {
        const int4 item = v.col_items[it];
        const int cell0 = item.x - (item.w >> 4);  // the column's first; the item's are at most kColumnSpan
        const int slot0 = v.cell_start[item.x], n = v.cell_start[item.x + (item.w & 15)] - slot0;
        const int groups = (n + 31) >> 5;
        double energy = 0.0;
        for (int g = item.y; g < groups; g += item.z) {
            const DevSpace &S = v.spaces[v.cell_rep[cell0]];
            const int per = n / groups, rest = n - per * groups;
            const int s0 = slot0 + g * per + min(g, rest), nown = per + (g < rest ? 1 : 0);
            const bool live = lane < nown;
            const float4 xi = live ? v.pos[s0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            ColOwn own;
            own.vel = (kKind != kTerms && live) ? v.vel[s0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            const int own_id = __float_as_int(own.vel.w);  // but for tables
            own.type = __float_as_int(xi.w);
            own.slot = s0 + lane;
            const int zi = live ? v.cell_of[s0 + lane] - cell0 : 0;
            const int zlo = __shfl_sync(kFull, zi, 0), zhi = __shfl_sync(kFull, zi, nown - 1);
            int loc[3];
            cell_loc(S, cell0, loc);
            const int cz = S.cdim[2];
            const float unit = S.col_unit, scale = S.col_scale;  // 2^26 to 2^27 units a cell edge
            const int edge = __float2int_rn(S.h[2] * scale);  // a cell edge (the cells are cubic)
            const float far = 7.f * S.h[2];
            const int zmid = (zhi - zlo + 1) * (edge >> 1) + edge;  // of the staged cells, one below zlo on
            own.zrel = zi - zlo;
            own.x = __float2int_rn(xi.x * scale) - (edge >> 1);
            own.y = __float2int_rn(xi.y * scale) - (edge >> 1);
            own.z = column_z(__float2int_rn(xi.z * scale), zi - zlo + 1, edge, -zmid);
            // pairs within a rounding of the cutoff, of their potential's a or of a table's end go to odd_pairs
            const float cut2 = S.cut2_pair * scale * scale * (1.f + S.near_cut), cut2_in = S.cut2_pair * scale * scale * (1.f - S.near_cut);
            float blo[3], bhi[3], reach2;
            {
                const float p[3] = {(float)own.x, (float)own.y, (float)own.z};
                // the candidate test's expanded squares round at the size of the warp's cells
                const float ef = (float)edge, ez = (float)zmid;
                reach2 = fmaxf(S.cut2w_pair, S.cut2w_self) * scale * scale + 2e-6f * (4.5f * ef * ef + ez * ez);
                __syncwarp();
                sm.own_xy[lane] = make_ulonglong2(pack2(-2.f * p[0], -2.f * p[0]), pack2(-2.f * p[1], -2.f * p[1]));
                const float side = on_grid(xi, far) ? reach2 - __fmaf_rn(p[0], p[0], __fmaf_rn(p[1], p[1], p[2] * p[2]))
                                                    : __int_as_float(0xff800000);
                sm.own_zr[lane] = make_ulonglong2(pack2(-2.f * p[2], -2.f * p[2]), pack2(side, 0.f));
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int q = k == 0 ? own.x : k == 1 ? own.y : own.z;
                    blo[k] = (float)__reduce_min_sync(kFull, live ? q : 0x7fffffff);
                    bhi[k] = (float)__reduce_max_sync(kFull, live ? q : (int)0x80000000);
                }
            }
            // particles near a face or outside their cells: some pairs may not be in reach of the task list
            bool careful = S.off_cell;
            if (S.prune & 2) {
                bool near = false;
                for (int k = lane; k <= zhi - zlo; k += 32) near |= v.cell_near[cell0 + zlo + k] != 0;
                if (__any_sync(kFull, near)) careful |= any_skipped(v, S, loc[0], loc[1], zlo, zhi);
            }
            // ---- runs of slots: lane 3 p + q < 9 the column (p - 1, q - 1) within a cell of the warp's z
            // range, 9 and 18 lanes on its cells beyond the lower and the upper z face
            __syncwarp();
            int cnt = 0;
            int4 run = make_int4(0, 0, 0, 0), off = make_int4(0, 0, 0, 0);
            if (lane < 27) {
                const int col9 = lane % 9, which = lane / 9;
                int nx = loc[0] + col9 / 3 - 1, ny = loc[1] + col9 % 3 - 1;
                bool there = true;
                // the shifts as the task list has them (across a periodic face, rounded at the box's size)
                float sx = S.sh[0], sy = S.sh[1];
                if (nx < 0 || nx >= S.cdim[0]) {
                    there = there && (S.periodic & 1);
                    nx += nx < 0 ? S.cdim[0] : -S.cdim[0];
                    sx = S.shw[0];
                }
                if (ny < 0 || ny >= S.cdim[1]) {
                    there = there && (S.periodic & 2);
                    ny += ny < 0 ? S.cdim[1] : -S.cdim[1];
                    sy = S.shw[1];
                }
                off.x = (col9 / 3 - 1) * __float2int_rn(sx * scale) - (edge >> 1);
                off.y = (col9 % 3 - 1) * __float2int_rn(sy * scale) - (edge >> 1);
                off.z = -zmid + (which == 0 ? 0 : (which == 1 ? -1 : 1) * (__float2int_rn(S.shw[2] * scale) - edge));
                int za = max(zlo - 1, 0), zb = min(zhi + 1, cz - 1);
                if (which == 1) {
                    za = zb = cz - 1;
                    there = there && zlo == 0 && (S.periodic & 4);
                } else if (which == 2) {
                    za = zb = 0;
                    there = there && zhi == cz - 1 && (S.periodic & 4);
                }
                if (there) {
                    const int col = S.cell_offset + (nx * S.cdim[1] + ny) * cz;
                    run.x = v.cell_start[col + za];
                    cnt = v.cell_start[col + zb + 1] - run.x;
                    // cell - run.z: the staged particle's z cell, one up from the cell below zlo
                    run.z = col + zlo - 1 + (which == 1 ? cz : which == 2 ? -cz : 0);
                }
                run.w = lane;
            }
            int incl = cnt;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(kFull, incl, off);
                if (lane >= off) incl += o;
            }
            if (lane < 27) {
                run.x -= incl - cnt;  // slot = run.x + index
                run.y = incl;
                sm.run[lane] = run;
                sm.off[lane] = off;
            }
            const int total = __shfl_sync(kFull, incl, 31);
            __syncwarp();
            // with one type the pair's constants stay in registers
            const bool one_type = ntypes == 1;
            constexpr int kBatch = needs_velocities(kKind) ? 3 : 2;  // rounds of 32 loaded together: more cost registers
            const int pair_base = S.pot_offset + own.type * ntypes;
            const unsigned rng_mode = S.rng_mode;
            const float near2 = v.near_dpd * (scale * scale);
            const double inv_cutoff = 1.0 / S.cutoff_d;
            float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
            if (kKind == kTermsPureDpd && one_type) {
                q0 = __ldg(v.dpd_pair + 2 * S.pot_offset);
                q1 = __ldg(v.dpd_pair + 2 * S.pot_offset + 1);
            }
            PairRec rec;
            rec.p = rec.q = q0;
            if (kKind == kTermsFlux) {
                const bool first = live && w == 0;  // the carried rates, once
                for (int k = 0; k < 8; ++k)
                    sm.rate[k][lane] = first && k < sp.smax ? sp.rate[(size_t)own_id * sp.smax + k] : 0.f;
            }
            if ((kKind == kTerms || kKind == kTermsDpd) && one_type) rec = load_rec(v.pair_rec, S.pot_offset);
            float3 f = make_float3(0.f, 0.f, 0.f);
            // this warp's rounds: of every 64 particles the 32 with even places, then, from the start again,
            // those with odd ones. The halves are alike in space, so when a region holds one of them a
            // lane's neighbours are shared out evenly between the regions
            const int evens = (((total + 63) >> 6) + kSplit - 1 - w) / kSplit, rounds = 2 * evens;
            int m0 = 0, rk = 0;
#pragma unroll 1
            while (m0 < rounds) {
                // ---- staging: batches of kBatch x 32 while another one fits
                int base = 0;
                sm.self[lane] = -1;
                __syncwarp();
#pragma unroll 1
                while (m0 < rounds && base <= Smem::kCap - 32) {
                    const int batch = min(kBatch, min(rounds - m0, (Smem::kCap - base) >> 5));
                    float4 q[kBatch];
                    int slot[kBatch], zq[kBatch], cq[kBatch];
#pragma unroll
                    for (int r = 0; r < kBatch; ++r) {
                        const int round = m0 + r;
                        const int odd = round >= evens;
                        const int idx = ((odd ? round - evens : round) * kSplit + w) * 64 + 2 * lane + odd;
                        slot[r] = -1;
                        if (r < batch && round == evens) rk = 0;
                        if (r < batch && idx < total) {
                            while (idx >= sm.run[rk].y) ++rk;
                            const int4 rr = sm.run[rk];
                            slot[r] = rr.x + idx;
                            cq[r] = rr.w;
                            q[r] = v.pos[slot[r]];
                            zq[r] = v.cell_of[slot[r]] - rr.z;
                        }
                    }
                    m0 += batch;
#pragma unroll
                    for (int r = 0; r < kBatch; ++r) {
                        bool keep = false;
                        int4 b;
                        if (slot[r] >= 0) {
                            const int4 o = sm.off[cq[r]];
                            b.x = __float2int_rn(q[r].x * scale) + o.x;
                            b.y = __float2int_rn(q[r].y * scale) + o.y;
                            b.z = column_z(__float2int_rn(q[r].z * scale), zq[r], edge, o.z);
                            b.w = zq[r] << 11 | cq[r] << 6 | __float_as_int(q[r].w);
                            // distance to the box of the warp's own particles
                            const float px = (float)b.x, py = (float)b.y, pz = (float)b.z;
                            const float ex = fmaxf(fmaxf(blo[0] - px, px - bhi[0]), 0.f);
                            const float ey = fmaxf(fmaxf(blo[1] - py, py - bhi[1]), 0.f);
                            const float ez = fmaxf(fmaxf(blo[2] - pz, pz - bhi[2]), 0.f);
                            keep = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, ez * ez)) <= reach2 && on_grid(q[r], far);
                        }
                        const unsigned bal = __ballot_sync(kFull, keep);
                        if (keep) {
                            const int at = base + __popc(bal & lt_mask);
                            sm.nb[at] = b;
                            if (needs_velocities(kKind)) cp_async16(&sm.nb_v[at], v.vel + slot[r]);
                            if (kKind != kTermsPureDpd)
                                sm.slot[at] = kKind == kTermsFlux ? __float_as_int(v.vel[slot[r]].w) : slot[r];
                            if (cq[r] == 4 && (unsigned)(slot[r] - s0) < (unsigned)nown) sm.self[slot[r] - s0] = at;
                        }
                        base += __popc(bal);
                    }
                }
                if (needs_velocities(kKind)) cp_async_wait_all();
                if (lane == 0) {  // the place past the last
                    const int far = 0x40000000;
                    sm.nb[Smem::kCap] = make_int4(far, far, far, 0);
                    if (needs_velocities(kKind)) sm.nb_v[Smem::kCap] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                __syncwarp();
                // ---- candidates
                const int ngrp = (base + 31) >> 5;
                int u = 0;
                for (; u + 3 <= ngrp; u += 4) candidates<kKind, 2>(sm, u, base, nown);
                if (u < ngrp) candidates<kKind, 1>(sm, u, base, nown);
                const int me = sm.self[lane];  // not its own neighbour
                if (me >= 0) sm.mask[me >> 5][lane] &= ~(1u << (me & 31));
                if (careful) drop_unreached<kKind>(v, sm, S, loc[0], loc[1], zi, zi - zlo, ngrp, live);
                // ---- pairs: each lane walks its own bits, group by group over those that hold any
                unsigned some = 0u;
                int left = 0;
                for (u = 0; u < ngrp; ++u) {
                    const unsigned b = sm.mask[u][lane];
                    some |= b ? 1u << u : 0u;
                    left += __popc(b);
                }
                if (!live) {
                    left = 0;
                    some = 0u;
                }
                const int most = __reduce_max_sync(kFull, left);
                unsigned bits = 0u;
                int gbase = 0;
                bool odd = false;
                ColSums sum = {0.f, 0.f, 0.f, 0.0};  // of this region: shorter chains of FP32 additions
                unsigned long long sx = 0ull, sy = 0ull, sz = 0ull;  // two sums each, of every other pair
                // the next neighbour's staged index, or the place past the last, beyond any reach
                auto next = [&]() -> int {
                    if (bits == 0u && some) {
                        const int q = __ffs(some) - 1;
                        some &= some - 1u;
                        bits = sm.mask[q][lane];
                        sm.mask[q][lane] = 0u;
                        gbase = q * 32 - 1;
                    }
                    const int jj = bits ? gbase + __ffs(bits) : Smem::kCap;
                    bits &= bits - 1u;
                    return jj;
                };
                auto later = [&](int jj) {  // a pair for odd_pairs
                    sm.mask[jj >> 5][lane] |= 1u << (jj & 31);
                    odd = true;
                };
                // a pair's force is fs * (tx, ty, tz)
                auto pair = [&](int jj, float &fs, float &tx, float &ty, float &tz) {
                    const int4 b = sm.nb[jj];
                    const float dx = (float)(own.x - b.x), dy = (float)(own.y - b.y), dz = (float)(own.z - b.z);
                    const float s2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));  // r^2 in units^2
                    const bool within = s2 <= cut2;
                    fs = 0.f;
                    tx = dx;
                    ty = dy;
                    tz = dz;
                    if constexpr (kKind == kTermsFlux) {
                        if (!within) return;
                        const float r = fminf(__fsqrt_rn(s2) * unit, (float)S.cutoff_d);
                        const int c9 = ((b.w >> 6) & 31) % 9;
                        const int side = (c9 / 3 - 1) * 9 + (c9 % 3 - 1) * 3 + (b.w >> 11) - 1 - own.zrel;
                        const int id_j = sm.slot[jj];  // in a cell the lower slot is first, the lower id too
                        // the weight vanishes at the cutoff, a flux's decay does not
                        if (s2 > cut2_in && !reference_within(v, S, own.slot, v.slot_of_id[id_j], loc[0], loc[1], zi, c9,
                                                              (b.w >> 11) - 1 - own.zrel, side))
                            return;
                        pair_fluxes<kKind>(v, sp, sm, lane, own_id, own.type, id_j, b.w & 63, side > 0 || (side == 0 && own_id < id_j),
                                           r, inv_cutoff);
                        return;
                    } else if constexpr (kKind == kTermsPureDpd) {
                        if (!one_type) {
                            const int pk = pair_base + (b.w & 63);
                            q0 = __ldg(v.dpd_pair + 2 * pk);
                            q1 = __ldg(v.dpd_pair + 2 * pk + 1);
                        }
                        const float4 vj = sm.nb_v[jj];
                        const float ir = rsqrt_ftz(s2);
                        // zero beyond this pair's own cutoff (its constants are zero without a potential)
                        const float oc = fmaxf(__fmaf_rn(-__fmul_rn(s2, ir), q1.z * unit, 1.0f), 0.f);
                        const float dv = __fmaf_rn(dx, own.vel.x - vj.x, __fmaf_rn(dy, own.vel.y - vj.y, dz * (own.vel.z - vj.z)));
                        fs = dpd_term(oc, ir, dv, q0.z, q1.w);
                        // than a, or for the direction
                        const bool near = s2 < near2;
                        if (near && within) later(jj);
                        fs = within && !near ? fs : 0.f;
                    } else {
                        const int pk = pair_base + (b.w & 63);
                        if (!one_type) rec = load_rec(v.pair_rec, pk);
                        const float r2 = s2 * (unit * unit);
                        // from past a to before the table's end or the cutoff
                        bool use = r2 >= rec.p.x && (kKind == kTerms ? r2 <= rec.p.w : s2 <= cut2_in);
                        const bool met = kKind == kTerms ? r2 <= rec.p.w * v.near_ratio : within;
                        float e;
                        tx = dx * unit;
                        ty = dy * unit;
                        tz = dz * unit;
                        if (kKind == kTerms) {
                            const bool in = table_term(rec, v.coef, r2, e, fs) && use;
                            fs = in ? -fs : 0.f;
                            e = in ? e : 0.f;
                        } else {
                            fs = e = 0.f;
                            if (use) {
                                bool edge;
                                if (!pair_term(v, rec, tx, ty, tz, r2, own.vel, sm.nb_v[jj], rng_mode, fs, e, edge))
                                    fs = e = 0.f;
                                use = !edge;
                                if (v.pot_idx2) {  // a second potential summed on the pair
                                    const PairRec rec2 = load_rec(v.pair_rec2, pk);
                                    float f2 = 0.f, e2 = 0.f;
                                    if (rec2.code() != -2 && !(r2 < rec2.p.x - 2.f * v.near_r2)) {
                                        if (pair_term(v, rec2, tx, ty, tz, r2, own.vel, sm.nb_v[jj], rng_mode, f2, e2, edge)) {
                                            fs += f2;
                                            e += e2;
                                        }
                                        use = use && !edge && r2 >= rec2.p.x;
                                    }
                                }
                                if (!use) fs = e = 0.f;
                            }
                        }
                        if (met && !use) later(jj);
                        sum.e += (double)e;
                    }
                };
                // two neighbours at a time without branches between them, so that their loads and arithmetic
                // overlap
#pragma unroll 1
                for (int k = 0; k < most; k += 2) {
                    const int ja = next(), jb = next();
                    float fa, xa, ya, za, fb, xb, yb, zb;
                    pair(ja, fa, xa, ya, za);
                    pair(jb, fb, xb, yb, zb);
                    if (kKind != kTermsFlux) {
                        const unsigned long long f2 = pack2(fa, fb);
                        sx = fma2(f2, pack2(xa, xb), sx);
                        sy = fma2(f2, pack2(ya, yb), sy);
                        sz = fma2(f2, pack2(za, zb), sz);
                    }
                }
                if (kKind != kTermsFlux) {
                    const float2 px = unpack2(sx), py = unpack2(sy), pz = unpack2(sz);
                    sum.x = px.x + px.y;
                    sum.y = py.x + py.y;
                    sum.z = pz.x + pz.y;
                }
                if (kKind != kTermsFlux && __any_sync(kFull, odd)) {
                    const ColSums c = odd_pairs<kKind>(v, sm, S, own, loc[0], loc[1], zi, ngrp, live);
                    sum.x += c.x;
                    sum.y += c.y;
                    sum.z += c.z;
                    sum.e += c.e;
                }
                f.x += sum.x;
                f.y += sum.y;
                f.z += sum.z;
                energy += sum.e;
                __syncwarp();
            }
            if constexpr (kKind == kTermsFlux) {
                __syncwarp();
                if (kSplit > 1) __syncthreads();
                if (live && w == 0 && sp.nspec[own.type] > 0) {
                    for (int k = 0; k < sp.smax; ++k) {
                        float t = sm.rate[k][lane];
                        for (int q = 1; q < kSplit; ++q) t += reinterpret_cast<Smem *>(col_smem)[q].rate[k][lane];
                        sp.rate[(size_t)own_id * sp.smax + k] = t;
                    }
                }
                if (kSplit > 1) __syncthreads();
                continue;
            }
            if (kSplit > 1) {  // the warps' sums, in order
                float4 *share = reinterpret_cast<float4 *>(sm.own_xy);
                __syncwarp();
                share[lane] = make_float4(f.x, f.y, f.z, 0.f);
                __syncthreads();
                if (w == 0) {
#pragma unroll
                    for (int k = 1; k < kSplit; ++k) {
                        const float4 o = reinterpret_cast<const float4 *>(reinterpret_cast<Smem *>(col_smem)[k].own_xy)[lane];
                        f.x += o.x;
                        f.y += o.y;
                        f.z += o.z;
                    }
                }
                __syncthreads();
            }
            if (live && (kSplit == 1 || w == 0)) {
                // constant_force (MxForce.cpp:339-344), scale 1
                const DevType &T = v.types[own.type];
                v.force[s0 + lane] = T.has_force ? make_float4(T.fx + f.x, T.fy + f.y, T.fz + f.z, 0.f)
                                                 : make_float4(f.x, f.y, f.z, 0.f);
            }
        }
        // ---- the item's energy (DPD tabulates none): every pair was met from both sides. A row for each
        // warp of the widest split
        if (kKind == kTerms || kKind == kTermsDpd) {
            double e = 0.5 * energy;
            for (int off = 16; off > 0; off >>= 1) e += __shfl_xor_sync(kFull, e, off);
            double *row = v.epot_cell + v.nitems + kColumnParts * it;
            if (lane == 0) row[w] = e;
            if (w == 0 && lane >= kSplit && lane < kColumnParts) row[lane] = 0.0;
        }
    }
}

template <int kKind, int kSplit>
void configure_one() {
    cudaFuncSetAttribute(column_force_kernel<kKind, kSplit>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(ColSmem<kKind>) * kSplit);
    cudaFuncSetAttribute(column_force_kernel<kKind, kSplit>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
}

template <int kKind, int kSplit>
void launch_one(const EngineView &v, const SpeciesView &sp, int grid, cudaStream_t st) {
    const int blocks = std::max(1, std::min(grid, v.ncol_items));
    column_force_kernel<kKind, kSplit><<<blocks, 32 * kSplit, sizeof(ColSmem<kKind>) * kSplit, st>>>(v, sp);
}

template <int kKind>
void launch_kind(const EngineView &v, const SpeciesView &sp, int split, int grid, cudaStream_t st) {
    if (split >= 8)
        launch_one<kKind, 8>(v, sp, grid, st);
    else if (split >= 4)
        launch_one<kKind, 4>(v, sp, grid, st);
    else
        launch_one<kKind, 1>(v, sp, grid, st);
}

template <int kKind>
void configure_kind() {
    configure_one<kKind, 1>();
    configure_one<kKind, 4>();
    configure_one<kKind, 8>();
}

}  // namespace

void configure_column_kernels() {
    configure_kind<kTerms>();
    configure_kind<kTermsDpd>();
    configure_kind<kTermsPureDpd>();
    configure_kind<kTermsFlux>();
}

void launch_column_fluxes(const EngineView &v, const SpeciesView &sp, int split, cudaStream_t st) {
    if (v.ncol_items > 0) launch_kind<kTermsFlux>(v, sp, split, v.ncol_items, st);
}

void launch_column_force(const EngineView &v, bool has_dpd, int split, int grid, cudaStream_t st) {
    if (v.ncol_items == 0) return;
    const SpeciesView none{};
    if (has_dpd && v.dpd_pure == 1)
        launch_kind<kTermsPureDpd>(v, none, split, grid, st);
    else if (has_dpd || v.pot_idx2)
        launch_kind<kTermsDpd>(v, none, split, grid, st);
    else
        launch_kind<kTerms>(v, none, split, grid, st);
}

}  // namespace mxg

// SPH neighbour lists: one tree walk per step, exact lists per pass.
//
// The reference gets an i-group and a superset j-list from FDPS for every
// density, derivative and hydro call (TreeForForceShort::Gather / Symmetry,
// main.cpp:79-81, 139-143).  Here the j-sets are explicit: for particle i
//   gather    : { j : |x_j - x_i|^2 < (2.5 h_i)^2 }            (density, derivative)
//   symmetric : { j : |x_j - x_i|^2 < max(2.5 h_i, 2.5 h_j)^2 }  (hydro)
// in ascending key order, identical to the oracle's (oracle/sph_oracle.c:
// or_sph_walk).
//
// 1. Units: octree cells with at most 32 particles whose parent holds more;
//    consecutive sibling units are packed into one warp while they fit.
//    Units are spatially compact (inside one parent cell), so no warp sees
//    a group box that straddles a jump of the Morton curve.
// 2. Superset walk, once per step (after the sort): every warp walks the
//    octree depth-first in octant order with its unit's bounding box and
//    keeps j with r_ij < KAPPA * max(H_i, H_j) (FP32 with a generous margin),
//    the h of that moment being recorded as h_sup.
// 3. Per pass, a filter kernel keeps the exact set from the superset: FP32
//    on double-float coordinates with an error band of 2^-19 relative, the
//    exact FP64 test of the oracle inside the band.  The superset contains
//    the exact set as long as every h <= KAPPA * h_sup; the filter raises a
//    flag otherwise and the host rebuilds the superset with the current h.
#include <algorithm>
#include <cstring>

#include "sph_fixpoint.cuh"
#include "sph_physics.cuh"

namespace sph {

constexpr float KAPPA = 1.06f;   // measured at 1M: 1.15 -> 13.7 ms, 1.10 -> 12.9, 1.06 -> 12.6, 1.03 -> 13.0 (repairs)
// walk warps per block: one, so a block's SM slot is freed as soon as its walk unit is done (the
// units' walks differ in length); 1M walk: 1.95 ms with four warps per block, 1.97 with two,
// 1.92 with one (about 30 blocks per SM, limited by shared memory)
constexpr int NB_WARPS = 1;
constexpr int WALK_SMALL = 100, WALK_MID = 330;   // particles per SM below which 4 / 2 warps walk a unit
constexpr int DENS_SMALL = 200;   // particles per SM below which the density takes 8 threads per particle
constexpr int ROW_K_MAX = 512;   // widest row block; longer rows continue in spill ranges (RowMap)
constexpr int NB_SURV = 64;    // ring of culled candidates staged for the pair test
constexpr int NB_FREE = 16;    // stack entries beyond NB_STACK: room for the accepted entries of a batch at any depth
constexpr int NB_STACK = 264;   // depth-first from any stack of <= NB_MULTI entries: + 21 levels x 7 pending siblings + 1
constexpr int NB_MULTI = 116;   // the stack may reach this with several cells expanded at once
constexpr unsigned FULLM = 0xffffffffu;

__device__ __forceinline__ float df_sub(float ah, float al, float bh, float bl) { return (ah - bh) + (al - bl); }

// ---------------------------------------------------------------------------
// superset walk: one warp per unit

struct WalkTree {
    const int4 *cinfo;   // first_child, n_child, start, count
    const float4 *blo, *bhi;
};

__device__ __forceinline__ float gap2_rd(float4 a_lo, float4 a_hi, float3 glo, float3 ghi) {
    const float gx = fmaxf(0.0f, fmaxf(__fsub_rd(a_lo.x, ghi.x), __fsub_rd(glo.x, a_hi.x)));
    const float gy = fmaxf(0.0f, fmaxf(__fsub_rd(a_lo.y, ghi.y), __fsub_rd(glo.y, a_hi.y)));
    const float gz = fmaxf(0.0f, fmaxf(__fsub_rd(a_lo.z, ghi.z), __fsub_rd(glo.z, a_hi.z)));
    return __fadd_rd(__fadd_rd(__fmul_rd(gx, gx), __fmul_rd(gy, gy)), __fmul_rd(gz, gz));
}

// Bound by instruction issue (about three a cycle per SM with 32 one-warp blocks), so what is left is what the tests
// need: a step of the walk takes up to 32 leaves or four inner cells from one read of the stack's top, a candidate's
// place comes from a scan and a vote, pairs are tested two per instruction in full batches of 32 survivors, and an
// accepted pair's owner and survivor are read from a list that the lanes wrote instead of searched for.  1M particles:
// 1.71 -> 1.08 billion instructions, 1.92 -> 1.42 ms (the searches, leaves eight at a time by a loop, and tests one by
// one before); 100,000 0.32 -> 0.25 ms, 5,000 124 -> 109 us.
// SPILL: rows may continue in spill ranges (walks after this step's spill layout); without it
// the hot loop carries no spill code (a row longer than K only raises the overflow flag)
template <bool SPILL>
__global__ void __launch_bounds__(NB_WARPS * 32, 32 / NB_WARPS)
k_sup_walk(int n_units, int split, const int2 *__restrict__ units, const int *__restrict__ uidx, const double *__restrict__ x,
           const double *__restrict__ y, const double *__restrict__ z, const double *__restrict__ h,
           double *__restrict__ hsup, const float4 *__restrict__ xh,
           const float4 *__restrict__ xl, const float *__restrict__ H2f, const int *__restrict__ prun, WalkTree T,
           int *__restrict__ sup,
           float *__restrict__ sup_r2, float *__restrict__ sup_m, int *__restrict__ cnt, RowMap rm, int *uover,
           int *err, int *maxcnt) {
    // cells to visit: (first_child, -n_child) for an internal cell, (start, count) for a leaf
    __shared__ int2 s_stack[NB_WARPS][NB_STACK + NB_FREE];
    // candidates that survived the per-particle cull: index; hi x, y, z, mass, lo x, y, z, kappa'^2 (2.5 h_j)^2
    __shared__ int s_sj[NB_WARPS][NB_SURV];
    __shared__ __align__(16) float s_sv[NB_WARPS][8][NB_SURV];
    // every lane's double-float position, for the lanes that write another lane's entries
    __shared__ float4 s_pih[NB_WARPS][32], s_pil[NB_WARPS][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * NB_WARPS + warp;
    if (w >= n_units * split) return;   // warp-uniform
    const int uid = uidx ? uidx[w / split] : w / split;
    // this warp's part of the unit
    int2 U = units[uid];
    const int part = w % split, part_n = (U.y + split - 1) / split;
    const int parts = (U.y + part_n - 1) / part_n;   // non-empty parts
    U.x += part * part_n;
    U.y = min(U.y - part * part_n, part_n);
    if (U.y <= 0) return;   // warp-uniform
    const int K = rm.K;
    const bool valid = lane < U.y;
    const int i = U.x + (valid ? lane : 0);
    const double xi = x[i], yi = y[i], zi = z[i];
    if (hsup && valid) hsup[i] = h[i];   // the h this row is built for (null: it is built for the recorded one)
    const float4 pih = xh[i], pil = xl[i];
    const float H2i = valid ? H2f[i] : 0.0f;
    double lo[3] = {valid ? xi : INFINITY, valid ? yi : INFINITY, valid ? zi : INFINITY};
    double hi[3] = {valid ? xi : -INFINITY, valid ? yi : -INFINITY, valid ? zi : -INFINITY};
    float R2 = H2i;
    for (int o = 16; o > 0; o >>= 1) {
        for (int d = 0; d < 3; ++d) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(FULLM, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_xor_sync(FULLM, hi[d], o));
        }
        R2 = fmaxf(R2, __shfl_xor_sync(FULLM, R2, o));
    }
    const float3 glo = make_float3(__double2float_rd(lo[0]), __double2float_rd(lo[1]), __double2float_rd(lo[2]));
    const float3 ghi = make_float3(__double2float_ru(hi[0]), __double2float_ru(hi[1]), __double2float_ru(hi[2]));
    const float k2 = KAPPA * KAPPA * 1.00390625f;          // kappa^2 (1 + 2^-8): generous, only a superset is needed
    const float Rg = __fmul_ru(KAPPA * 1.00390625f, __fsqrt_ru(R2));
    const float Rg2 = __fmul_ru(Rg, Rg);
    const unsigned lt = (1u << lane) - 1u;
    int2 *stack = s_stack[warp];
    int *sj = s_sj[warp];
    float(*sv)[NB_SURV] = s_sv[warp];
    int count = 0;         // accepted entries of this lane's row
    int wr = 0, rd = 0;    // staged survivors, tested ones (a multiple of 32)
    int sp = 0;            // cells on the stack
    // the spill range continues a row at entry K: entry k >= K of particle p at
    // rm.main + rm.soff[p] - K + k (computed on the rare paths that need it)
    auto spill_cap = [&]() { return valid ? row_spill_cap(rm, i) : 0; };
    s_pih[warp][lane] = pih;
    s_pil[warp][lane] = pil;
    __syncwarp();

    // 32 staged survivors (the last batch: n of them) against every lane, without branching (bit t of `am`), two
    // survivors per instruction.  The accepted entries, lane by lane and in survivor order within a lane, are
    // numbered e = 0 .. total - 1, listed as (lane, survivor) in the free part of the stack's memory, and written by
    // the whole warp, 32 at a time: a lane's run of entries lands contiguously in its row, so every store covers a
    // few runs instead of 32 rows.
    const f32x2 nxh = f2_pack(-pih.x, -pih.x), nyh = f2_pack(-pih.y, -pih.y), nzh = f2_pack(-pih.z, -pih.z),
                nxl = f2_pack(-pil.x, -pil.x), nyl = f2_pack(-pil.y, -pil.y), nzl = f2_pack(-pil.z, -pil.z);
    const float ti = k2 * H2i;
    auto batch = [&](int n) {
        const int s0 = rd & (NB_SURV - 1);
        unsigned am = 0;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            if (4 * g >= n) break;
            auto four = [&](int c) { return *reinterpret_cast<const ulonglong2 *>(&sv[c][s0 + 4 * g]); };
            const ulonglong2 xh4 = four(0), yh4 = four(1), zh4 = four(2), xl4 = four(4), yl4 = four(5), zl4 = four(6);
            const float4 tj = *reinterpret_cast<const float4 *>(&sv[7][s0 + 4 * g]);
            auto r2_of = [&](f32x2 xh2, f32x2 yh2, f32x2 zh2, f32x2 xl2, f32x2 yl2, f32x2 zl2) {
                const f32x2 dx = f2_add(f2_add(xh2, nxh), f2_add(xl2, nxl));
                const f32x2 dy = f2_add(f2_add(yh2, nyh), f2_add(yl2, nyl));
                const f32x2 dz = f2_add(f2_add(zh2, nzh), f2_add(zl2, nzl));
                return f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
            };
            float ra, rb, rc, rd4;
            f2_unpack(r2_of(xh4.x, yh4.x, zh4.x, xl4.x, yl4.x, zl4.x), ra, rb);
            f2_unpack(r2_of(xh4.y, yh4.y, zh4.y, xl4.y, yl4.y, zl4.y), rc, rd4);
            if (ra < fmaxf(ti, tj.x)) am |= 1u << (4 * g);
            if (rb < fmaxf(ti, tj.y)) am |= 2u << (4 * g);
            if (rc < fmaxf(ti, tj.z)) am |= 4u << (4 * g);
            if (rd4 < fmaxf(ti, tj.w)) am |= 8u << (4 * g);
        }
        if (n < 32) am &= (1u << n) - 1u;
        if (!valid) am = 0u;
        const int nacc = __popc(am);
        int incl = nacc;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULLM, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(FULLM, incl, 31);
        const int before = count - (incl - nacc);   // entry e of this lane is entry before + e of its row
        unsigned short *ent = reinterpret_cast<unsigned short *>(stack + sp);
        const int room = 4 * (NB_STACK + NB_FREE - sp);
        for (int e0 = 0; e0 < total; e0 += room) {
            int e = incl - nacc - e0;
            for (unsigned x = am; x; x &= x - 1, ++e)
                if ((unsigned)e < (unsigned)room) ent[e] = (unsigned short)(lane << 5 | (__ffs(x) - 1));
            __syncwarp();
            const int m = min(total - e0, room);
            for (int q0 = 0; q0 < m; q0 += 32) {
                const int q = q0 + lane;
                const int le = q < m ? ent[q] : 0, L = le >> 5, t = s0 + (le & 31);
                const int pos = __shfl_sync(FULLM, before, L) + e0 + q;
                if (q < m) {
                    const float4 qh = s_pih[warp][L], ql = s_pil[warp][L];
                    const float dx = df_sub(sv[0][t], sv[4][t], qh.x, ql.x);
                    const float dy = df_sub(sv[1][t], sv[5][t], qh.y, ql.y);
                    const float dz = df_sub(sv[2][t], sv[6][t], qh.z, ql.z);
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    const int iL = U.x + L;
                    if (pos < K) {
                        const int64_t o = (int64_t)iL * K + pos;
                        sup[o] = sj[t];
                        sup_r2[o] = r2;
                        sup_m[o] = sv[3][t];
                    } else if (SPILL && pos < K + row_spill_cap(rm, iL)) {
                        const int64_t o = rm.main + rm.soff[iL] - K + pos;
                        sup[o] = sj[t];
                        sup_r2[o] = r2;
                        sup_m[o] = sv[3][t];
                    }
                }
            }
            __syncwarp();
        }
        count += nacc;
    };

    // Up to 32 candidates are culled, each against the unit's box grown by its own reach: a lower bound of the
    // distance (the point's hi / lo interval, rounded down) against an upper bound of max(Rg, kappa' 2.5 h_j), so no
    // pair the test above would accept is dropped.  Survivors are staged with their coordinates.
    auto cull = [&](int j, bool act) {
        bool keep = false;
        float4 qh = make_float4(0.f, 0.f, 0.f, 0.f), ql = qh;
        if (act) {
            qh = xh[j];
            ql = xl[j];
            ql.w = H2f[j];
            const float ex = fabsf(ql.x), ey = fabsf(ql.y), ez = fabsf(ql.z);
            const float gx = fmaxf(0.0f, fmaxf(__fsub_rd(__fsub_rd(qh.x, ex), ghi.x),
                                               __fsub_rd(glo.x, __fadd_ru(qh.x, ex))));
            const float gy = fmaxf(0.0f, fmaxf(__fsub_rd(__fsub_rd(qh.y, ey), ghi.y),
                                               __fsub_rd(glo.y, __fadd_ru(qh.y, ey))));
            const float gz = fmaxf(0.0f, fmaxf(__fsub_rd(__fsub_rd(qh.z, ez), ghi.z),
                                               __fsub_rd(glo.z, __fadd_ru(qh.z, ez))));
            const float g2 = __fadd_rd(__fadd_rd(__fmul_rd(gx, gx), __fmul_rd(gy, gy)), __fmul_rd(gz, gz));
            keep = g2 < fmaxf(Rg2, __fmul_ru(k2, ql.w));
        }
        const unsigned km = __ballot_sync(FULLM, keep);
        if (keep) {
            const int p = (wr + __popc(km & lt)) & (NB_SURV - 1);
            sj[p] = j;
            sv[0][p] = qh.x;
            sv[1][p] = qh.y;
            sv[2][p] = qh.z;
            sv[3][p] = qh.w;
            sv[4][p] = ql.x;
            sv[5][p] = ql.y;
            sv[6][p] = ql.z;
            sv[7][p] = k2 * ql.w;
        }
        wr += __popc(km);
        __syncwarp();
        if (wr - rd >= 32) {
            batch(32);
            rd += 32;
        }
    };

    {
        const int root = prun[U.x];   // the unit's run's octree root
        const float4 a = T.blo[root], b = T.bhi[root];
        const float R = fmaxf(Rg, __fmul_ru(2.5f * KAPPA * 1.00390625f, b.w));
        if (gap2_rd(a, b, glo, ghi) < __fmul_ru(R, R)) {
            if (lane == 0) {
                const int4 r = T.cinfo[root];
                stack[0] = r.y == 0 ? make_int2(r.z, r.w) : make_int2(r.x, -r.y);
            }
            sp = 1;
        }
        __syncwarp();
    }
    while (sp > 0) {
        const int2 se = lane < sp ? stack[sp - 1 - lane] : make_int2(0, 0);   // lane 0: the top
        const unsigned leaves = __ballot_sync(FULLM, se.y > 0);
        if (leaves & 1u) {   // a leaf: with the leaves right below it, while their particles fit 32 lanes
            const int run = leaves == FULLM ? 32 : __ffs(~leaves) - 1;
            const int v = lane < run ? min(se.y, 33) : 0;
            int incl = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(FULLM, incl, o);
                if (lane >= o) incl += u;
            }
            const int k = __popc(__ballot_sync(FULLM, lane < run && incl <= 32));
            if (k > 0) {
                // lane -> (leaf, offset): leaves in stack order from the top, particles in order
                const unsigned first = __reduce_or_sync(FULLM, lane < k ? 1u << (incl - v) : 0u);
                const int tot = __shfl_sync(FULLM, incl, k - 1);
                const int g = __popc(first & ((2u << lane) - 1u)) - 1;
                const int j = __shfl_sync(FULLM, se.x - (incl - v), g) + lane;
                sp -= k;
                cull(j, lane < tot);
            } else {   // a leaf above 32 particles (only at the deepest level)
                const int s = __shfl_sync(FULLM, se.x, 0), ct = __shfl_sync(FULLM, se.y, 0);
                --sp;
                for (int b0 = 0; b0 < ct; b0 += 32) cull(s + b0 + lane, b0 + lane < ct);
            }
        } else {
            // up to four internal cells from the top of the stack expanded at once, eight lanes per
            // cell: their children are pushed so that the top cell's come first, as the one-cell
            // expansion would visit them (the leaves, and so the rows, keep their order).  More
            // than one only while the stack stays below NB_MULTI, so a depth-first continuation
            // (at most 7 pending siblings per level below) still fits NB_STACK.
            const int inner = leaves ? __ffs(leaves) - 1 : 32;
            const int k = min(min(4, sp), min(inner, max(1, (NB_MULTI - sp) / 7)));
            const int g = lane >> 3, q = lane & 7;
            const int f = __shfl_sync(FULLM, se.x, g), nch = -__shfl_sync(FULLM, se.y, g);
            bool ok = false;
            int2 chi = make_int2(0, 0);
            if (g < k && q < nch) {
                const float4 a = T.blo[f + q], b = T.bhi[f + q];
                const int4 r = T.cinfo[f + q];   // independent of the box loads: one round trip
                chi = r.y == 0 ? make_int2(r.z, r.w) : make_int2(r.x, -r.y);
                const float R = fmaxf(Rg, __fmul_ru(2.5f * KAPPA * 1.00390625f, b.w));
                ok = gap2_rd(a, b, glo, ghi) < __fmul_ru(R, R);
            }
            sp -= k;
            __syncwarp();
            const unsigned mask = __ballot_sync(FULLM, ok);
            const int np = __popc(mask);
            if (sp + np > NB_STACK) {
                if (lane == 0) atomicOr(err, ERR_SPH_STACK);
                break;
            }
            if (ok) stack[sp + (np - 1 - __popc(mask & ((1u << lane) - 1u)))] = chi;
            sp += np;
            __syncwarp();
        }
    }
    if (wr > rd) batch(wr - rd);
    if (valid) {
        const int scap = (SPILL && count > K) ? spill_cap() : 0;
        cnt[i] = count;   // the true count, also when the row had no room for all of it
        if (count > K + scap) atomicOr(err, ERR_SPH_LIST_OVERFLOW);
    }
    int m = valid ? count : 0;
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(FULLM, m, o));
    if (lane == 0) {
        atomicMax(maxcnt, m);
        // the unit holds rows that need a spill range: one bit per part
        if (split == 1) uover[uid] = m > K ? 1 : 0;
        else if (m > K) atomicOr(&uover[uid], 1 << part);
        else atomicAnd(&uover[uid], ~(1 << part));
        if (part == 0) atomicAnd(&uover[uid], (1 << parts) - 1);   // bits of parts this unit does not have
    }
}

// ---------------------------------------------------------------------------
// incremental repair after h outgrew the skin
//
// Every row i is built with the reach KAPPA max(2.5 hsup_i, 2.5 hsup_j), hsup
// being the h recorded when all rows were walked, so it holds all neighbours
// as long as h <= KAPPA hsup everywhere.  A particle v that violates this
// (or nears it) gets hsup_v = h_v, and the rows of every unit within
// KAPPA 2.5 h_v of it (its own among them) are walked again with that reach;
// hsup of all others stays.  Were the h of the moment used for the others,
// rows inside and outside the repaired units would hold different reaches for
// one particle: a larger one recorded is missing outside (a later growth
// inside the skin would not be seen there), a smaller one is missing inside.
//
// That is the FP64 passes' rule.  The mixed passes still repair by the h of the moment, within 2.5 h_v.  In a mixed step
// only violators change their h after a repair, so what can be missing is a violator that grows on, inside its new skin,
// from the row of a particle between 1 / KAPPA and 1 of its support away (found: one pair in 40 runs of 2,000 to 300,000
// particles, a few in 8 steps of 1M; a caller of single passes can see the other two cases too).  Such a pair weighs less
// than 1e-6 of the kernel's centre, but one entry more shifts the blocks of 32 that a row's FP32 partial sums are rounded
// in: with the FP64 rule 6 of 18 runs of 1M and 4M particles changed in last bits (up to 2e-7 of a component's
// rms; 4e-6 after 16 steps of a sweep), and a mixed run gives the same bits in every build so far.
//
// Between the FP64 density passes every h is still on its way, and a particle that has used most of its skin tends to
// leave it a pass later; so a repair takes in all that grew by more than SKIN_64, for fewer repairs in a row (prologue
// of 71,184 particles in contact 3 -> 2, of 10,000 2 -> 1; 53.1 -> 52.5 and 9.85 -> 9.76 ms with four steps).
constexpr double SKIN_64 = 1.04;

// vR: reach (`reach` times 2.5 h) of the particles a repair takes in (h > grown hsup; 0: the others); nviol: the violators
// among them
__global__ void k_viol_mark(int n, double grown, double reach, const double *h, const double *hsup, float *vR,
                            int *nviol) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool v = false;
    if (i < n) {
        v = h[i] > (double)KAPPA * hsup[i];
        vR[i] = h[i] > grown * hsup[i] ? __double2float_ru(SUPPORT * h[i] * reach) : 0.0f;
    }
    const unsigned b = __ballot_sync(FULLM, v);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(nviol, __popc(b));
}

// what a repair's walk is built for: hsup raised to h for the particles it takes in, (2.5 hsup)^2 as k_h2f
__global__ void k_skin_raise(int n, const double *h, const float *vR, double *hsup, float *H2s) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double s = vR[i] > 0.0f ? h[i] : hsup[i];
    hsup[i] = s;
    const double H = SUPPORT * s;
    H2s[i] = __double2float_ru(H * H);
}

// after a density round: (2.5 h)^2 of the new h as k_h2f, and the count of k_viol_mark
__global__ void k_h2f_viol(int n, const double *h, const double *hsup, float *H2f, int *nviol) {
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool v = false;
    if (i < n) {
        const double H = SUPPORT * h[i];
        H2f[i] = __double2float_ru(H * H);
        v = h[i] > (double)KAPPA * hsup[i];
    }
    const unsigned b = __ballot_sync(FULLM, v);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(nviol, __popc(b));
}

__global__ void k_cell_vmax(int l, const int *meta, const float *vR, const int4 *cinfo, float *cvR) {
    const int L0 = meta[l], L1 = meta[l + 1];
    for (int c = L0 + blockIdx.x * blockDim.x + threadIdx.x; c < L1; c += gridDim.x * blockDim.x) {
        const int4 ci = cinfo[c];
        float r = 0.0f;
        if (ci.y == 0) {
            for (int j = ci.z; j < ci.z + ci.w; ++j) r = fmaxf(r, vR[j]);
        } else {
            for (int k = 0; k < ci.y; ++k) r = fmaxf(r, cvR[ci.x + k]);
        }
        cvR[c] = r;
    }
}

// warp per unit: is any violator within its reach of the unit's box?
__global__ void __launch_bounds__(NB_WARPS * 32)
k_unit_mark(int n_units, const int2 *__restrict__ units, const float4 *__restrict__ xh, const float4 *__restrict__ xl,
            const float *__restrict__ vR, const float *__restrict__ cvR, const int4 *__restrict__ cinfo,
            const float4 *__restrict__ blo, const float4 *__restrict__ bhi, const int *__restrict__ prun,
            int *umark) {
    __shared__ int s_stack[NB_WARPS][NB_STACK];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = blockIdx.x * NB_WARPS + warp;
    if (u >= n_units) return;
    const int2 U = units[u];
    const bool valid = lane < U.y;
    const int i = U.x + (valid ? lane : 0);
    const float4 ph = xh[i], pl = xl[i];
    // unit box in float, widened by one ulp each way (the double-float sum rounds)
    float lo[3] = {valid ? ph.x + pl.x : INFINITY, valid ? ph.y + pl.y : INFINITY, valid ? ph.z + pl.z : INFINITY};
    float hi[3] = {valid ? ph.x + pl.x : -INFINITY, valid ? ph.y + pl.y : -INFINITY,
                   valid ? ph.z + pl.z : -INFINITY};
    for (int o = 16; o > 0; o >>= 1)
        for (int d = 0; d < 3; ++d) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(FULLM, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(FULLM, hi[d], o));
        }
    const float3 glo = make_float3(nextafterf(lo[0], -INFINITY), nextafterf(lo[1], -INFINITY),
                                   nextafterf(lo[2], -INFINITY));
    const float3 ghi = make_float3(nextafterf(hi[0], INFINITY), nextafterf(hi[1], INFINITY),
                                   nextafterf(hi[2], INFINITY));
    int *stack = s_stack[warp];
    int sp = 0;
    bool hit = false;
    {
        const int root = prun[U.x];   // the unit's run's octree root
        const float r = cvR[root];
        if (r > 0.0f && gap2_rd(blo[root], bhi[root], glo, ghi) < __fmul_ru(r, r)) {
            if (lane == 0) stack[0] = root;
            sp = 1;
        }
        __syncwarp();
    }
    while (sp > 0 && !hit) {
        const int c = stack[--sp];
        __syncwarp();
        const int4 ci = cinfo[c];
        if (ci.y == 0) {
            bool h2 = false;
            for (int j = ci.z + lane; j < ci.z + ci.w; j += 32) {
                const float r = vR[j];
                if (r > 0.0f) {
                    const float4 qh = xh[j], ql = xl[j];
                    const float px = qh.x + ql.x, py = qh.y + ql.y, pz = qh.z + ql.z;
                    const float4 a = make_float4(nextafterf(px, -INFINITY), nextafterf(py, -INFINITY),
                                                 nextafterf(pz, -INFINITY), 0.0f);
                    const float4 b = make_float4(nextafterf(px, INFINITY), nextafterf(py, INFINITY),
                                                 nextafterf(pz, INFINITY), 0.0f);
                    if (gap2_rd(a, b, glo, ghi) < __fmul_ru(r, r)) h2 = true;
                }
            }
            hit = __any_sync(FULLM, h2);
        } else {
            bool ok = false;
            int ch = 0;
            if (lane < ci.y) {
                ch = ci.x + lane;
                const float r = cvR[ch];
                ok = r > 0.0f && gap2_rd(blo[ch], bhi[ch], glo, ghi) < __fmul_ru(r, r);
            }
            const unsigned mask = __ballot_sync(FULLM, ok);
            const int np = __popc(mask);
            if (sp + np > NB_STACK) {   // cannot happen for an octree of depth 21; be safe: mark
                hit = true;
                break;
            }
            if (ok) stack[sp + (np - 1 - __popc(mask & ((1u << lane) - 1u)))] = ch;
            sp += np;
            __syncwarp();
        }
    }
    if (lane == 0) umark[u] = hit ? 1 : 0;
}

__global__ void k_unit_flag(int n_units, const int *uover, int *umark) {
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n_units; u += gridDim.x * blockDim.x)
        umark[u] = uover[u] != 0;
}

__global__ void k_unit_compact(int n_units, const int *umark, const int *off, int *uidx) {
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n_units; u += gridDim.x * blockDim.x)
        if (umark[u]) uidx[off[u]] = u;
}

// ---------------------------------------------------------------------------
// exact filter

// The FP32 r^2 stored by the walk is (x_j - x_i)^2 on double-float
// coordinates, within 2^-21 of the exact value; outside a band of 2^-19
// around the threshold it decides alone, inside it the oracle's FP64 test
// decides.
__device__ __forceinline__ bool exact_in(float r2, float thr, int j, double xi, double yi, double zi, double H2,
                                         const double *__restrict__ x, const double *__restrict__ y,
                                         const double *__restrict__ z, const double *__restrict__ h, bool sym) {
    if (r2 < thr * (1.0f - 1.9073486328125e-06f)) return true;
    if (r2 > thr * (1.0f + 1.9073486328125e-06f)) return false;
    const double ex = __dsub_rn(x[j], xi), ey = __dsub_rn(y[j], yi), ez = __dsub_rn(z[j], zi);
    const double rr = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
    if (rr < H2) return true;
    if (sym) {
        const double Hj = __dmul_rn(SUPPORT, h[j]);
        return rr < __dmul_rn(Hj, Hj);
    }
    return false;
}

// the same with the i-particle's doubles loaded only inside the band
__device__ __forceinline__ bool exact_in(float r2, float thr, int j, int i, const double *__restrict__ x,
                                         const double *__restrict__ y, const double *__restrict__ z,
                                         const double *__restrict__ h, bool sym) {
    if (r2 < thr * (1.0f - 1.9073486328125e-06f)) return true;
    if (r2 > thr * (1.0f + 1.9073486328125e-06f)) return false;
    const double Hi = __dmul_rn(SUPPORT, h[i]);
    return exact_in(r2, thr, j, x[i], y[i], z[i], __dmul_rn(Hi, Hi), x, y, z, h, sym);
}

// exact_in behind a call: a loop that decides several entries before summing them would
// otherwise have the FP64 test if-converted, issuing its FP64 instructions for every entry
__device__ __noinline__ bool exact_in_call(float r2, float thr, int j, double xi, double yi, double zi, double H2,
                                           const double *__restrict__ x, const double *__restrict__ y,
                                           const double *__restrict__ z, const double *__restrict__ h) {
    return exact_in(r2, thr, j, xi, yi, zi, H2, x, y, z, h, false);
}

// MODE 0: gather list, 1: symmetric list, 2: both (the gather set is a subset of the symmetric set, so its test runs
// only on symmetric members).  Bound by the latency of the dependent loads (entry, then h of its particle) and by the
// bytes of the superset rows.  A warp per row: 32 entries at a time, loads and compacted stores contiguous, entries
// loaded two chunks and h one chunk ahead, 16 blocks per SM at 32 registers (12 blocks: 0.64 ms at 1M, 10:
// 0.73); outside the edge band nothing touches the FP64 pipe, (2.5 h_i)^2 coming from the rounded-up float copy
// (within the band the exact test decides, whatever the copy's rounding).  One thread per row, eight entries at a time, took 0.87 ms at 1M and 84 us at 5,003 particles; a warp takes 0.57 ms and 27 us.
constexpr int FW = 4;   // rows (warps) per block
constexpr float BAND_LO = 1.0f - 1.9073486328125e-06f, BAND_HI = 1.0f + 1.9073486328125e-06f;   // exact_in's band

// entry k of a row: in the row block, or (SPILL rows, k >= K) in its spill range, base + k
template <bool SPILL, class T>
__device__ __forceinline__ T *entry(T *blk, T *spill, int K, int k) {
    return (SPILL && k >= K ? spill : blk) + k;
}

template <int MODE, bool SPILL>
__device__ __forceinline__ void filter_row(int i, int lane, int c, int K, int64_t spill, const int *__restrict__ sup,
                                           const float *__restrict__ sup_r2, const double *__restrict__ x,
                                           const double *__restrict__ y, const double *__restrict__ z,
                                           const double *__restrict__ h, const float *__restrict__ H2f, int *out0,
                                           int *out1, int &k0, int &k1) {
    const int64_t blk = (int64_t)i * K;
    const int *row = sup + blk, *row_s = sup + spill;
    const float *rrow = sup_r2 + blk, *rrow_s = sup_r2 + spill;
    int *o0 = out0 + blk, *o0_s = out0 + spill, *o1 = out1 + blk, *o1_s = out1 + spill;
    const unsigned lt = (1u << lane) - 1u;
    const float H2i = H2f[i], lo0 = H2i * BAND_LO, hi0 = H2i * BAND_HI;
    // two chunks ahead: entries; one chunk ahead: the h of their particles
    int jn = i, jm = i;
    // past the end: a NaN is below no threshold and inside no band, not even where 2.5 h squared overflows to infinity
    const float none = __int_as_float(0x7fffffff);
    float rn = none, rm = none;
    if (lane < c) {
        jn = *entry<SPILL>(row, row_s, K, lane);
        rn = *entry<SPILL>(rrow, rrow_s, K, lane);
    }
    if (lane + 32 < c) {
        jm = *entry<SPILL>(row, row_s, K, lane + 32);
        rm = *entry<SPILL>(rrow, rrow_s, K, lane + 32);
    }
    float hn = MODE != 0 ? H2f[jn] : 0.0f;
    for (int b = 0; b < c; b += 32) {
        const int j = jn, kn = b + 64 + lane;
        const float r2 = rn, hj = hn;
        jn = jm;
        rn = rm;
        if (MODE != 0) hn = H2f[jn];
        rm = none;
        if (kn < c) {
            jm = *entry<SPILL>(row, row_s, K, kn);
            rm = *entry<SPILL>(rrow, rrow_s, K, kn);
        }
        bool in0 = r2 < lo0, edge0 = !in0 && r2 <= hi0, in1 = false, edge1 = false;
        if (MODE != 0) {
            const float t = fmaxf(H2i, hj);
            in1 = r2 < t * BAND_LO;
            edge1 = !in1 && r2 <= t * BAND_HI;
        }
        if (__any_sync(FULLM, (MODE != 1 && edge0) || edge1)) {   // rare: the exact test decides
            if (edge1) in1 = exact_in(r2, fmaxf(H2i, hj), j, i, x, y, z, h, true);
            if (MODE != 1 && edge0) in0 = exact_in(r2, H2i, j, i, x, y, z, h, false);
        }
        if (MODE != 1) {
            const unsigned m = __ballot_sync(FULLM, in0);
            if (in0) *entry<SPILL>(o0, o0_s, K, k0 + __popc(m & lt)) = j;
            k0 += __popc(m);
        }
        if (MODE != 0) {
            const unsigned m = __ballot_sync(FULLM, in1);
            if (in1) *entry<SPILL>(o1, o1_s, K, k1 + __popc(m & lt)) = j;
            k1 += __popc(m);
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(FW * 32, 16)
k_filter(int n, const int *__restrict__ sup, const float *__restrict__ sup_r2, const int *__restrict__ scnt,
         RowMap rm, const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
         const double *__restrict__ h, const float *__restrict__ H2f, int *__restrict__ out0, int *__restrict__ ocnt0,
         int *__restrict__ out1, int *__restrict__ ocnt1) {
    const int lane = threadIdx.x & 31, i = blockIdx.x * FW + (threadIdx.x >> 5);
    if (i >= n) return;   // warp-uniform
    const int c = scnt[i], K = rm.K;
    int k0 = 0, k1 = 0;
    if (c <= K)
        filter_row<MODE, false>(i, lane, c, K, 0, sup, sup_r2, x, y, z, h, H2f, out0, out1, k0, k1);
    else
        filter_row<MODE, true>(i, lane, c, K, rm.main + rm.soff[i] - K, sup, sup_r2, x, y, z, h, H2f, out0, out1, k0,
                               k1);
    if (lane == 0) {
        if (MODE != 1) ocnt0[i] = k0;
        if (MODE != 0) ocnt1[i] = k1;
    }
}

// Every density pass of a step (CalcDensity, force.h:9-23, main.cpp:138-139) for a particle
// in one go: the passes only use the particle's own h, and its row holds its gather set as
// long as h <= KAPPA h_sup.  DT threads share a particle (entries 4 sub .. 4 sub + 3 in steps
// of 4 DT; 8 for small runs, whose passes are the latency of
// one thread's chain: 5,000 particles 36 -> 19 us, 20,000 41 -> 34, equal at 40,000; measured at 1M: DT 1 1.07 ms, 2 0.98, 4 0.97 for the four passes before the loop
// below was made branch-free); a particle whose new h leaves the skin stops after that pass, to
// go on once its row is walked again.  The four entries of a chunk are decided first (the rare
// FP64 edge test behind a call), then summed without branches, two at a time in paired FP32
// arithmetic, non-members as zero terms (0.98 -> 0.69 ms at 1M, bit-identical).  Each term
// m_j W_ij is rounded to a multiple of 2^-40 and summed as an integer, so the sum depends on
// neither the order of the terms nor where non-members sit in the row.  The multiple is taken on
// the particle's run's own mass scale (the terms carry the context's, 2^fixd[run] times the
// run's: a power of two), so a run's sums are the same alone and in any mix of runs.  SPLIT:
// every run's masses on its own scale are at most 15, so each term is at most 16 and takes
// sph_fix40_add (FP32 / integer pipes) instead of __float2ll_rn (FP64 pipe); both give the same
// integers.  Blocks of 64 threads (32 particles): 0.67 -> 0.65 ms at 1M against 128.
template <bool SPLIT, int DT>
__global__ void __launch_bounds__(64)
k_density_fused32(int n, int n_pass, const int *__restrict__ sup, const float *__restrict__ sup_r2,
                  const float *__restrict__ sup_m, const int *__restrict__ scnt, RowMap rm,
                  const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
                  const double *__restrict__ m, double *__restrict__ h, const double *__restrict__ hsup,
                  double *__restrict__ dens, float dscale, int *__restrict__ npass, int *n_stopped,
                  const int *__restrict__ prun, const int *__restrict__ fixd) {
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = gt / DT, sub = gt % DT;
    if (i >= n) return;   // whole groups leave together
    int p = npass[i];
    if (p >= n_pass) return;
    // the fixed-point grid 2^(fd - 40) on the context's scale is 2^-40 on the run's
    // (powers of two written as bit patterns: exponent fields moved by fd, |fd| <= 60)
    const int fd = fixd[prun[i]];
    const unsigned b1 = SPH_FIX_B1 + ((unsigned)fd << 23), b2 = SPH_FIX_B2 + ((unsigned)fd << 23);
    const float c1 = __uint_as_float(b1), c2 = __uint_as_float(b2);
    const float to_fix = __uint_as_float((unsigned)(127 + 40 - fd) << 23);                         // 2^(40 - fd)
    const double from_fix = __longlong_as_double((long long)(1023 + fd - 40) << 52);               // 2^(fd - 40)
    const unsigned gm = __activemask();
    double hi = h[i];
    const double hs = hsup[i], xi = x[i], yi = y[i], zi = z[i], mi = m[i];
    const int c_all = scnt[i];
    bool stopped = false;
    for (; p < n_pass && !stopped; ++p) {
        const double Hi = __dmul_rn(SUPPORT, hi);
        const double H2 = __dmul_rn(Hi, Hi);
        const float H2i = (float)H2;
        const float invH = 1.0f / (float)Hi;
        const float lo_b = H2i * (1.0f - 1.9073486328125e-06f), hi_b = H2i * (1.0f + 1.9073486328125e-06f);
        long long acc = 0;
        // SPLIT: 32-bit sums of the raw bit patterns of sph_fix40_add's a and b, their offsets
        // (b1, b2 per term, non-members included: a zero term adds exactly the offsets) taken off
        // when they are flushed, after at most SPH_FIX_TERMS terms
        unsigned rH = 0, rL = 0, nt = 0;   // nt: terms in rH / rL
        const f32x2 ih2 = f2_pack(invH, invH), one2 = f2_pack(1.0f, 1.0f), c1_2 = f2_pack(c1, c1),
                    c2_2 = f2_pack(c2, c2), k32 = f2_pack(32.0f, 32.0f), k25 = f2_pack(25.0f, 25.0f),
                    k8 = f2_pack(8.0f, 8.0f);
        for (int seg = 0; seg < 2; ++seg) {
            int c;
            const int64_t b = row_seg(rm, i, seg, c_all, &c);
            if (c <= 0) break;
            const float *rrow = sup_r2 + b, *mrow = sup_m + b;
            // the next chunk's r^2 loads while this chunk is summed (1M, four passes: 0.69 -> 0.67
            // ms; r^2 and m both ahead: 0.68 ms, more registers)
            float4 rn = 4 * sub < c ? *reinterpret_cast<const float4 *>(rrow + 4 * sub) : make_float4(0.f, 0.f, 0.f, 0.f);
            for (int k = 4 * sub; k < c; k += 4 * DT) {
                if (SPLIT) {
                    if (nt == (unsigned)SPH_FIX_TERMS) {
                        acc += sph_fix40_value(rH - nt * b1, rL - nt * b2);
                        rH = rL = nt = 0;
                    }
                    nt += 4;
                }
                const float4 r4 = rn;
                const float4 m4 = *reinterpret_cast<const float4 *>(mrow + k);
                if (k + 4 * DT < c) rn = *reinterpret_cast<const float4 *>(rrow + k + 4 * DT);
                const float rr[4] = {r4.x, r4.y, r4.z, r4.w};
                // members: inside the band by FP32, at its edge by the FP64 test; padding out
                bool in[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    in[u] = k + u < c && rr[u] < lo_b;
                    if (k + u < c && !in[u] && !(rr[u] > hi_b))
                        in[u] = exact_in_call(rr[u], H2i, sup[b + k + u], xi, yi, zi, H2, x, y, z, h);
                }
                // m_j W(s) for two entries at a time, each lane with the roundings of the scalar
                // m * ((1 + s (8 + s (25 + 32 s))) (q^4 q^4)), q = max(1 - s, 0), s = sqrt(r^2) / H
                float t[4];
#pragma unroll
                for (int pr = 0; pr < 2; ++pr) {
                    const f32x2 s2 = f2_mul(f2_pack(sqrt_a(rr[2 * pr]), sqrt_a(rr[2 * pr + 1])), ih2);
                    float qa, qb;
                    f2_unpack(f2_sub(one2, s2), qa, qb);
                    const f32x2 q = f2_pack(fmaxf(qa, 0.0f), fmaxf(qb, 0.0f));
                    const f32x2 q2 = f2_mul(q, q), q4 = f2_mul(q2, q2);
                    const f32x2 poly = f2_fma(s2, f2_fma(s2, f2_fma(s2, k32, k25), k8), one2);
                    const f32x2 mj = pr == 0 ? f2_pack(m4.x, m4.y) : f2_pack(m4.z, m4.w);
                    f2_unpack(f2_mul(mj, f2_mul(poly, f2_mul(q4, q4))), t[2 * pr], t[2 * pr + 1]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) t[u] = in[u] ? t[u] : 0.0f;
                if (SPLIT) {
#pragma unroll
                    for (int pr = 0; pr < 2; ++pr) {
                        const f32x2 tt = f2_pack(t[2 * pr], t[2 * pr + 1]);
                        const f32x2 a = f2_add(tt, c1_2);
                        const f32x2 bb = f2_add(f2_sub(tt, f2_sub(a, c1_2)), c2_2);
                        float a0, a1, b0, b1f;
                        f2_unpack(a, a0, a1);
                        f2_unpack(bb, b0, b1f);
                        rH += __float_as_uint(a0) + __float_as_uint(a1);
                        rL += __float_as_uint(b0) + __float_as_uint(b1f);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc += __float2ll_rn(t[u] * to_fix);
                }
            }
        }
        if (SPLIT) acc += sph_fix40_value(rH - nt * b1, rL - nt * b2);
#pragma unroll
        for (int o = DT / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(gm, acc, o, DT);
        double rho, hn;
        density_tail32((float)((double)acc * from_fix), invH, dscale, mi, &rho, &hn);
        hi = hn;
        if (sub == 0) {
            dens[i] = rho;
            h[i] = hn;
        }
        // the row can miss members of the next pass's set: the same test as k_viol_mark
        stopped = p + 1 < n_pass && hn > (double)KAPPA * hs;
    }
    if (sub == 0) {
        npass[i] = p;
        if (stopped) atomicAdd(n_stopped, 1);
    }
}

// (2.5 h)^2 as float, rounded up so FP32 superset tests stay conservative
__global__ void k_h2f(int n, const double *h, float *H2f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double H = SUPPORT * h[i];
    H2f[i] = __double2float_ru(H * H);
}

// double-float positions (hi / lo floats); .w of xh carries the mass x mscale; (2.5 h)^2 as k_h2f
__global__ void k_pack_pos(int n, const double *x, const double *y, const double *z, const double *m, double mscale,
                           const double *h, float4 *xh, float4 *xl, float *H2f) {
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double H = SUPPORT * h[i];
    H2f[i] = __double2float_ru(H * H);
    float a, b, c, d, e, f;
    split_df(x[i], a, d);
    split_df(y[i], b, e);
    split_df(z[i], c, f);
    xh[i] = make_float4(a, b, c, (float)(m[i] * mscale));
    xl[i] = make_float4(d, e, f, 0.0f);
}

// spill range lengths: rows longer than K take round8(count - K) entries beyond the row block
__global__ void k_spill_need(int n, const int *cnt, int K, int *need, unsigned long long *total) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int v = 0;
    if (i < n) v = cnt[i] > K ? ((cnt[i] - K + 7) & ~7) : 0;
    if (i <= n) need[i] = v;
    // the sum in 64 bits: the offsets are 32-bit, so a total past 2^31 must be refused, not wrapped
    unsigned long long w = (unsigned long long)v;
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(total, w);
}

}  // namespace sph

using namespace sph;

template <class T>
static int dalloc_n(sph_ctx *ctx, T **p, int64_t n) {
    if (*p) cudaFree(*p);
    *p = nullptr;
    cudaError_t e = cudaMalloc((void **)p, sizeof(T) * (size_t)std::max<int64_t>(n, 1));
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return sph_fail(ctx, SPH_ERR_OOM, "device allocation of %lld bytes failed", (long long)(sizeof(T) * n));
    }
    return SPH_OK;
}

// the double-float positions the walks read: in the mixed path the packs of sph_pack_mixed
// (written after every sort, before any walk, with the same split and the same mass in .w),
// in the FP64 path the walk's own
static const float4 *walk_xh(const sph_ctx *ctx) {
    return ctx->cfg.precision == SPH_PREC_MIXED ? ctx->xh : ctx->sup.pxh;
}
static const float4 *walk_xl(const sph_ctx *ctx) {
    return ctx->cfg.precision == SPH_PREC_MIXED ? ctx->xl : ctx->sup.pxl;
}

// h-dependent float copies; called after every density pass
int sph_nbr_refresh_h(sph_ctx *ctx) {
    SphSuper &S = ctx->sup;
    const int n = (int)ctx->n;
    k_h2f<<<sph_div_up(n, 256), 256, 0, ctx->stream>>>(n, FLD(ctx->F, SPH_SMTH, ctx->cap), S.H2f);
    ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    return SPH_OK;
}

// after the sort: positions as double-float, h as float, and the superset marked stale
int sph_nbr_prepare(sph_ctx *ctx) {
    SphSuper &S = ctx->sup;
    const int n = (int)ctx->n;
    const int64_t pitch = ((int64_t)n + 31) / 32 * 32;
    if (S.cap_particles < pitch) {
        SPH_TRY(dalloc_n(ctx, &S.pxh, pitch));
        SPH_TRY(dalloc_n(ctx, &S.pxl, pitch));
        SPH_TRY(dalloc_n(ctx, &S.H2f, pitch));
        SPH_TRY(dalloc_n(ctx, &S.H2s, pitch));
        SPH_TRY(dalloc_n(ctx, &S.hsup, pitch));
        SPH_TRY(dalloc_n(ctx, &S.cnt, pitch));
        SPH_TRY(dalloc_n(ctx, &S.vR, pitch));
        SPH_TRY(dalloc_n(ctx, &S.npass, pitch));
        S.cap_particles = pitch;
    }
    if (S.cap_cells < ctx->tree.cap) {
        S.cap_cells = ctx->tree.cap;
        SPH_TRY(dalloc_n(ctx, &S.cvR, S.cap_cells));
    }
    const int64_t cap = ctx->cap;
    if (ctx->cfg.precision == SPH_PREC_MIXED) {   // the mixed path walks on its own packs
        SPH_TRY(sph_pack_mixed(ctx));
    } else {
        launch_after(true, k_pack_pos, sph_div_up(n, 256), 256, 0, ctx->stream, n, FLD(ctx->F, SPH_X, cap),
                     FLD(ctx->F, SPH_Y, cap), FLD(ctx->F, SPH_Z, cap), FLD(ctx->F, SPH_MASS, cap), ctx->mscale,
                     FLD(ctx->F, SPH_SMTH, cap), S.pxh, S.pxl, S.H2f);
        ++ctx->launches;
    }
    SPH_CUDA(ctx, cudaGetLastError());
    S.valid = false;
    S.rebuilds_step = 0;
    ctx->lists[0].valid = ctx->lists[1].valid = false;
    return SPH_OK;
}

// walks the units in uidx (or all units when uidx is null) for the current h, which hsup records, or (recorded) for the
// hsup there is (k_skin_raise); grows the row capacity if needed
static int walk_units(sph_ctx *ctx, const int *uidx, int n_walk, bool recorded) {
    SphSuper &S = ctx->sup;
    const int n = (int)ctx->n;
    const int64_t pitch = n;   // rows: particle i's entries at i * K .. i * K + K - 1
    const int64_t cap = ctx->cap;
    int *meta = ctx->tree.meta;
    Tree &t = ctx->tree;
    if (S.K == 0) S.K = 192;
    S.K = (S.K + 7) & ~7;   // rows start on 32-byte boundaries
    if (!S.uover || S.n_units > S.cap_uover) {
        SPH_TRY(dalloc_n(ctx, &S.uover, S.cap_units));
        SPH_CUDA(ctx, cudaMemsetAsync(S.uover, 0, sizeof(int) * S.cap_units, ctx->stream));
        S.cap_uover = S.cap_units;
    }
    // cell hmax must follow the h that is walked for
    if (S.rebuilds_step > 0) SPH_TRY(sph_tree_refresh_hmax(ctx, recorded ? S.hsup : FLD(ctx->F, SPH_SMTH, cap)));
    S.rebuilds_step += 1;
    for (int attempt = 0; attempt < 4; ++attempt) {
        if (!S.nbr || S.pitch < pitch || S.K_alloc != S.K || S.spill_alloc != S.spill_cap) {
            if (uidx) {   // a partial walk cannot re-layout the rows: the others would be lost
                uidx = nullptr;
                n_walk = S.n_units;
            }
            if (S.K_alloc != S.K || S.pitch < pitch) S.spill_on = false;   // spill offsets follow K and n
            S.main = (int64_t)S.K * pitch;
            const int64_t tot = S.main + S.spill_cap;
            SPH_TRY(dalloc_n(ctx, &S.nbr, tot));
            SPH_TRY(dalloc_n(ctx, &S.r2, tot));
            SPH_TRY(dalloc_n(ctx, &S.m, tot));
            for (int m = 0; m < 2; ++m) {
                SPH_TRY(dalloc_n(ctx, &ctx->lists[m].nbr, tot));
                SPH_TRY(dalloc_n(ctx, &ctx->lists[m].cnt, pitch));
                ctx->lists[m].K = ctx->lists[m].K_alloc = S.K;
                ctx->lists[m].pitch = S.K;   // row stride of the exact lists
            }
            S.pitch = pitch;
            S.K_alloc = S.K;
            S.spill_alloc = S.spill_cap;
        }
        static_assert(META_MAXCNT == META_ERR + 1, "cleared together");
        if (attempt > 0 || S.rebuilds_step > 1)   // the first walk after a sort finds them cleared
            SPH_CUDA(ctx, cudaMemsetAsync(meta + META_ERR, 0, 2 * sizeof(int), ctx->stream));
        // A warp walks a unit, or two or four share it: the walk of a small run is the latency of one warp's chain
        // (depth-first steps, candidates, accepted entries), and more and shorter chains fill the chip.  Rows do not
        // depend on the split, and units stay the units of the skin repairs.  Walk of 5,000 / 10,000 particles by
        // one warp per unit 150 / 185 us, two 122 / 142, four 109 / 129; of 20,000 179, 141, 145; of 40,000 195, 172,
        // 199; 70,000 particles and more are fastest with one (214, 251, 301).
        const int64_t per_sm = n / ctx->num_sms;
        const int split = per_sm < WALK_SMALL ? 4 : (per_sm < WALK_MID ? 2 : 1);
        const int blocks = (n_walk * split + NB_WARPS - 1) / NB_WARPS;
        WalkTree T{t.cinfo, t.blo, t.bhi};
        if (blocks > 0) {
            auto walk = S.spill_on ? k_sup_walk<true> : k_sup_walk<false>;
            walk<<<blocks, NB_WARPS * 32, 0, ctx->stream>>>(n_walk, split, S.units, uidx, FLD(ctx->F, SPH_X, cap), FLD(ctx->F, SPH_Y, cap), FLD(ctx->F, SPH_Z, cap),
                FLD(ctx->F, SPH_SMTH, cap), recorded ? nullptr : S.hsup, walk_xh(ctx), walk_xl(ctx),
                recorded ? S.H2s : S.H2f, ctx->runs.prun, T, S.nbr, S.r2, S.m,
                S.cnt, S.map(), S.uover, meta + META_ERR, meta + META_MAXCNT);
            ++ctx->launches;
        }
        SPH_CUDA(ctx, cudaGetLastError());
        int *hs = (int *)ctx->host_scalars;
        SPH_TRY(sph_publish(ctx, meta + META_ERR, 2));
        SPH_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        const int errw = hs[0], maxc = hs[META_MAXCNT - META_ERR];
        if (errw & ERR_SPH_STACK) return sph_fail(ctx, SPH_ERR_CAPACITY, "SPH walk stack overflow");
        if (errw & ERR_SPH_LIST_OVERFLOW) {
            if (maxc <= ROW_K_MAX && !S.spill_on) {
                // every row fits a wider block: grow K and rebuild everything
                S.K = std::min(ROW_K_MAX, (maxc + maxc / 4 + 16 + 7) & ~7);
                uidx = nullptr;
                n_walk = S.n_units;
                continue;
            }
            // rows longer than K (the true counts are in cnt) get spill ranges; the units holding
            // them are walked again (all of them if the spill block had to grow)
            if (!S.soff || S.cap_soff < n + 1) {
                SPH_TRY(dalloc_n(ctx, &S.soff, n + 1 + 1024));
                SPH_TRY(dalloc_n(ctx, &S.need, n + 1 + 1024));
                S.cap_soff = n + 1 + 1024;
            }
            unsigned long long *tot64 = reinterpret_cast<unsigned long long *>(ctx->scratch_d);
            SPH_CUDA(ctx, cudaMemsetAsync(tot64, 0, sizeof(unsigned long long), ctx->stream));
            k_spill_need<<<sph_div_up(n + 1, 256), 256, 0, ctx->stream>>>(n, S.cnt, S.K, S.need, tot64);
            ++ctx->launches;
            SPH_CUDA(ctx, cudaMemcpyAsync(&ctx->host_scalars[1], tot64, sizeof(unsigned long long),
                                          cudaMemcpyDeviceToHost, ctx->stream));
            SPH_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            unsigned long long need64 = 0;
            std::memcpy(&need64, &ctx->host_scalars[1], sizeof(need64));
            if (need64 > (unsigned long long)INT32_MAX - 4096)
                return sph_fail(ctx, SPH_ERR_CAPACITY,
                                "neighbour rows need %llu entries beyond the row block (smoothing lengths out of "
                                "range?)", need64);
            SPH_TRY(sph_scan_exclusive(ctx, S.need, S.soff, nullptr, n + 1, ctx->scan.total));
            const int64_t need = (int64_t)need64;
            S.spill_on = true;
            S.spilled = need;
            if (need > S.spill_cap) {
                S.spill_cap = need + need / 2 + 4096;   // reallocated at the top of the loop, rows rebuilt
                continue;
            }
            const int grid = 2 * ctx->num_sms;
            k_unit_flag<<<grid, 256, 0, ctx->stream>>>(S.n_units, S.uover, S.umark);
            ++ctx->launches;
            SPH_TRY(sph_scan_exclusive(ctx, S.umark, S.uoff, nullptr, S.n_units, ctx->scan.total));
            k_unit_compact<<<grid, 256, 0, ctx->stream>>>(S.n_units, S.umark, S.uoff, S.uidx);
            ++ctx->launches;
            SPH_CUDA(ctx, cudaMemcpyAsync(hs, ctx->scan.total, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
            SPH_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            uidx = S.uidx;
            n_walk = hs[0];
            continue;
        }
        S.valid = true;
        if (uidx) S.repairs += 1;
        else S.rebuilds += 1;
        S.units_walked += n_walk;
        return SPH_OK;
    }
    return sph_fail(ctx, SPH_ERR_CAPACITY, "SPH superset capacity could not be grown");
}

// a full walk after a sort: the previous spill layout belongs to the previous order
static int build_superset(sph_ctx *ctx) {
    ctx->sup.spill_on = false;
    return walk_units(ctx, nullptr, ctx->sup.n_units, false);
}

// makes the superset valid for the current h: full walk after a sort, otherwise a repair of
// the units within reach of particles whose h outgrew the skin
static int ensure_superset(sph_ctx *ctx) {
    SphSuper &S = ctx->sup;
    if (!S.valid) return build_superset(ctx);
    const int n = (int)ctx->n;
    const int64_t cap = ctx->cap;
    int *meta = ctx->tree.meta;
    Tree &t = ctx->tree;
    float *vR = S.vR;
    SPH_CUDA(ctx, cudaMemsetAsync(meta + META_ERR + 8, 0, sizeof(int), ctx->stream));
    const bool exact = ctx->cfg.precision != SPH_PREC_MIXED;   // (see above)
    const double grown = exact ? SKIN_64 : (double)KAPPA, reach = exact ? KAPPA * 1.001 : 1.001;
    k_viol_mark<<<sph_div_up(n, 256), 256, 0, ctx->stream>>>(n, grown, reach, FLD(ctx->F, SPH_SMTH, cap), S.hsup, vR,
                                                              meta + META_ERR + 8);
    ++ctx->launches;
    int *hs = (int *)ctx->host_scalars;
    SPH_TRY(sph_publish(ctx, meta + META_ERR + 8, 1));
    SPH_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const int nviol = hs[0];
    if (nviol == 0) return SPH_OK;
    S.violators += nviol;
    if ((int64_t)nviol * 8 > n) return build_superset(ctx);   // widespread growth: walk everything
    if (exact) {
        k_skin_raise<<<sph_div_up(n, 256), 256, 0, ctx->stream>>>(n, FLD(ctx->F, SPH_SMTH, cap), vR, S.hsup, S.H2s);
        ++ctx->launches;
    }
    // influence radius per cell, bottom-up
    const int grid = 2 * ctx->num_sms;
    for (int l = t.depth; l >= 0; --l) {
        k_cell_vmax<<<grid, 128, 0, ctx->stream>>>(l, meta, vR, t.cinfo, S.cvR);
        ++ctx->launches;
    }
    const int blocks = (S.n_units + NB_WARPS - 1) / NB_WARPS;
    k_unit_mark<<<blocks, NB_WARPS * 32, 0, ctx->stream>>>(S.n_units, S.units, walk_xh(ctx), walk_xl(ctx), vR, S.cvR,
                                                           t.cinfo, t.blo, t.bhi, ctx->runs.prun, S.umark);
    ++ctx->launches;
    SPH_TRY(sph_scan_exclusive(ctx, S.umark, S.uoff, nullptr, S.n_units, ctx->scan.total));
    k_unit_compact<<<grid, 256, 0, ctx->stream>>>(S.n_units, S.umark, S.uoff, S.uidx);
    ++ctx->launches;
    SPH_TRY(sph_publish(ctx, ctx->scan.total, 1));
    SPH_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const int nmark = hs[0];
    return walk_units(ctx, S.uidx, nmark, exact);
}

// exact list of `mode` (0 gather, 1 symmetric, 2 both) from a superset that is valid for the current h
static int filter_lists(sph_ctx *ctx, int mode) {
    SphSuper &S = ctx->sup;
    const int n = (int)ctx->n;
    const int64_t cap = ctx->cap;
    SphLists &L0 = ctx->lists[0], &L1 = ctx->lists[1];
    auto filter = mode == 0 ? k_filter<0> : (mode == 1 ? k_filter<1> : k_filter<2>);
    filter<<<sph_div_up(n, FW), FW * 32, 0, ctx->stream>>>(n, S.nbr, S.r2, S.cnt, S.map(), FLD(ctx->F, SPH_X, cap), FLD(ctx->F, SPH_Y, cap), FLD(ctx->F, SPH_Z, cap),
        FLD(ctx->F, SPH_SMTH, cap), S.H2f, L0.nbr, L0.cnt, L1.nbr, L1.cnt);
    ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    if (mode != 1) L0.valid = true;
    if (mode != 0) L1.valid = true;
    return SPH_OK;
}

// the same, with the superset made valid first
int sph_build_sph_lists(sph_ctx *ctx, int mode) {
    SPH_TRY(ensure_superset(ctx));
    return filter_lists(ctx, mode);
}

// All density passes of the mixed path, the EoS and the exact lists of the final h: rounds of k_density_fused32, the
// rows of the particles that left their skin walked again between rounds (each round takes every unfinished particle
// at least one pass further, so there are at most n_dens_iter rounds).  The host has to know whether a particle
// stopped (another round) or outgrew its skin in the last pass (a repair before the lists); both are rare, so the EoS
// and the lists are launched behind the round before it knows, and run again where it was needed: they only read what
// the round wrote.  The wait for the answer was a gap in a small run's step, and the lists had one of their own:
// a step of 5,000 particles 473 -> 455 us, of 100,000 1.276 -> 1.239 ms.  While a download follows the step, the lists wait, so that what the EoS finished is sent first.
int sph_density_fused(sph_ctx *ctx) {
    SphSuper &S = ctx->sup;
    const int n = (int)ctx->n;
    const int64_t cap = ctx->cap;
    const int np = ctx->cfg.n_dens_iter;
    int *nviol = ctx->tree.meta + META_ERR + 8, *stopped = nviol + 1;
    int *hs = (int *)ctx->host_scalars;
    const bool ahead = !ctx->dl_host;
    for (int round = 0; round <= np; ++round) {
        SPH_TRY(ensure_superset(ctx));
        SPH_TRY(time_mark(ctx, SEG_DENS_LIST));
        if (round > 0) SPH_CUDA(ctx, cudaMemsetAsync(nviol, 0, 2 * sizeof(int), ctx->stream));   // else cleared by the tree
        const int dt = (int64_t)n < (int64_t)ctx->num_sms * DENS_SMALL ? 8 : 2;
        auto kd = ctx->runs.fix_split ? (dt == 8 ? k_density_fused32<true, 8> : k_density_fused32<true, 2>)
                                      : (dt == 8 ? k_density_fused32<false, 8> : k_density_fused32<false, 2>);
        kd<<<sph_div_up((int64_t)n * dt, 64), 64, 0, ctx->stream>>>(n, np, S.nbr, S.r2, S.m, S.cnt, S.map(), FLD(ctx->F, SPH_X, cap), FLD(ctx->F, SPH_Y, cap),
            FLD(ctx->F, SPH_Z, cap), FLD(ctx->F, SPH_MASS, cap), FLD(ctx->F, SPH_SMTH, cap), S.hsup,
            FLD(ctx->F, SPH_DENS, cap), (float)(1365.0 / 64.0 / (3.141592653589793 * ctx->mscale)), S.npass,
            stopped, ctx->runs.prun, ctx->runs.fixd);
        ++ctx->launches;
        launch_after(true, k_h2f_viol, sph_div_up(n, 256), 256, 0, ctx->stream, n, FLD(ctx->F, SPH_SMTH, cap), S.hsup,
                     S.H2f, nviol);
        ++ctx->launches;
        SPH_CUDA(ctx, cudaGetLastError());
        SPH_TRY(time_mark(ctx, SEG_DENS));
        SPH_TRY(sph_publish(ctx, nviol, 2));
        SPH_CUDA(ctx, cudaEventRecord(ctx->tree_done, ctx->stream));
        SPH_TRY(sph_pass_eos(ctx));
        SPH_TRY(time_mark(ctx, SEG_EOS));
        if (ahead) SPH_TRY(filter_lists(ctx, 2));
        SPH_CUDA(ctx, cudaEventSynchronize(ctx->tree_done));
        if (hs[1] == 0) break;
        ctx->lists[0].valid = ctx->lists[1].valid = false;
        if (round == np) return sph_fail(ctx, SPH_ERR_STATE, "density passes did not converge over the skin repairs");
    }
    const bool outgrown = hs[0] > 0;
    // final from here on
    SPH_TRY(dl_milestone(ctx, 1ull << SPH_DENS | 1ull << SPH_SMTH | 1ull << SPH_PRES | 1ull << SPH_SNDS));
    if (outgrown) SPH_TRY(ensure_superset(ctx));
    return outgrown || !ahead ? filter_lists(ctx, 2) : SPH_OK;
}

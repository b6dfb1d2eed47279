// Gravity interaction lists on the device (the SPH neighbour lists are in
// sph_nbr.cu).
//
// Gravity (TreeForForceLong::Monopole, main.cpp:83,90): one block per i-group
// (cells with <= n_group particles whose parent holds more) walks the tree
// with the group's FP64 bounding box; a child is opened iff
// dmin^2(box, com) <= (side / theta)^2.  Opened leaves give EPJ particle
// ranges, unopened children of opened cells give SPJ monopoles, in the
// breadth-first order of the oracle's or_grav_walk.  Counting pass, scan,
// filling pass.
#include <algorithm>
#include <climits>

#include "sph_physics.cuh"

namespace sph {

constexpr unsigned FULL = 0xffffffffu;


// --------------------------------------------------------------------------
// interaction lists of the gravity i-groups (found with the tree)

constexpr int GL_T = 128;      // threads per block: one i-group
constexpr int GLCAP = 2048;    // ring buffer of opened cells (power of two)

// Breadth-first walk, GL_T / 4 opened cells per iteration (four lanes each, children k and k + 4 per lane).
// Order (shared with the oracle's or_grav_walk): cells are opened in FIFO
// order starting at the root; an opened leaf appends its particles to EPJ;
// an opened internal cell appends its unopened children to SPJ and its
// opened children to the queue, both in octant order.
//
// Bound by the latency of the iterations (queue, cell record, centre of mass, test) and, in FP64, by the tests.  A
// warp per group with four cells per iteration took 76 iterations for the 300 cells a group opens, and 10,000
// particles are 134 warps for 152 SMs; a block per group takes a tenth of the iterations.  The distance test runs in
// FP32 on coordinates relative to the group's box centre with a bound on its error, the FP64 test deciding inside
// the bound.  Groups and both passes of
// 10,000 / 200,003 particles: 0.39 / 0.64 -> 0.16 / 0.32 ms.
template <bool FILL>
__global__ void __launch_bounds__(GL_T)
k_grav_lists(int ng, const int *__restrict__ group_cell, const double *__restrict__ x,
             const double *__restrict__ y, const double *__restrict__ z, const int4 *__restrict__ cinfo,
             const int *__restrict__ clevel, const double4 *__restrict__ com, const double *__restrict__ rb_all,
             const int *__restrict__ prun, int *n_epj, int *n_spj, const int *off_epj, const int *off_spj, int *epj,
             int *spj, int *err) {
    constexpr int GW = GL_T / 32;
    __shared__ int s_q[GLCAP];
    __shared__ double s_box[6];          // the group's box
    __shared__ double s_rb[MAX_LEVELS];  // opening radii squared
    __shared__ int s_w[2][GW][3];        // per warp: leaf particles, far children, near children
    const int g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int4 gi = cinfo[group_cell[g]];
    const int s = gi.z, cnt = gi.w;
    const int root = prun[s];   // the group's run: its octree root and opening radii
    const double *rb = rb_all + (int64_t)root * RB_STRIDE;
    if (tid < MAX_LEVELS) s_rb[tid] = rb[8 + tid];
    if (warp == 0) {   // minima and maxima on the integer images of the doubles (off the FP64 pipe)
        const double *p[3] = {x + s, y + s, z + s};
        for (int d = 0; d < 3; ++d) {
            long long lo = LLONG_MAX, hi = LLONG_MIN;
            for (int k = lane; k < cnt; k += 32) {
                const long long v = dorder_key(p[d][k]);
                lo = min(lo, v);
                hi = max(hi, v);
            }
            for (int o = 16; o > 0; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(FULL, lo, o));
                hi = max(hi, __shfl_xor_sync(FULL, hi, o));
            }
            if (lane == 0) {
                s_box[d] = dorder_value(lo);
                s_box[3 + d] = dorder_value(hi);
            }
        }
    }
    if (tid == 0) s_q[0] = root;
    __syncthreads();
    // the box's centre and half-widths in FP32 (rounded up), for the fast test
    double ctr[3];
    float half[3];
    for (int d = 0; d < 3; ++d) {
        ctr[d] = 0.5 * (s_box[d] + s_box[3 + d]);
        half[d] = __double2float_ru(fmax(s_box[3 + d] - ctr[d], ctr[d] - s_box[d]));
    }
    int ne = 0, ns = 0;
    const int be = FILL ? off_epj[g] : 0, bs = FILL ? off_spj[g] : 0;
    int head = 0, tail = 1;
    const int q = tid >> 2, k = tid & 3, qw = lane >> 2;
    const unsigned cellm = 0xFu << (qw * 4), before = (1u << (qw * 4)) - 1u;
    for (int it = 0; head < tail; ++it) {
        const int nproc = min(GL_T / 4, tail - head);
        const bool act = q < nproc;
        const int c = act ? s_q[(head + q) & (GLCAP - 1)] : 0;
        const int4 ci = act ? cinfo[c] : make_int4(0, 0, 0, 0);   // first_child, n_child, start, count
        const bool leaf = act && ci.y == 0;
        const int lc = leaf ? ci.w : 0;   // the same in the four lanes of a cell
        bool near[2] = {false, false}, far[2] = {false, false};
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int kk = k + 4 * hh;
            if (!(act && kk < ci.y)) continue;
            const int ch = ci.x + kk;
            const double4 cm = com[ch];
            const double p[3] = {cm.x, cm.y, cm.z};
            const double r2 = s_rb[clevel[ch]];
            // |com - centre| minus the half-width, each within 2^-21 of its terms; d2 between lo2 and hi2
            float d2 = 0.0f, e2 = 0.0f;
            for (int d = 0; d < 3; ++d) {
                const float a = fabsf((float)(p[d] - ctr[d])), dd = fmaxf(a - half[d], 0.0f);
                const float ed = 4.76837158203125e-07f * (a + half[d]);   // 2^-21
                d2 = fmaf(dd, dd, d2);
                e2 = fmaf(2.0f * dd + ed, ed, e2);
            }
            const float rf = (float)r2;
            bool nr;
            if (fabsf(d2 - rf) > e2 + 9.5367431640625e-07f * (d2 + rf)) {   // 2^-20: the sums and the rounding of r2
                nr = d2 <= rf;
            } else {   // (and where FP32 overflows: the comparison above is false for a NaN)
                double dd[3];
                for (int d = 0; d < 3; ++d) {
                    const double lo = s_box[d], hi = s_box[3 + d];
                    dd[d] = (p[d] < lo) ? __dsub_rn(lo, p[d]) : ((p[d] > hi) ? __dsub_rn(p[d], hi) : 0.0);
                }
                nr = __dadd_rn(__dadd_rn(__dmul_rn(dd[0], dd[0]), __dmul_rn(dd[1], dd[1])), __dmul_rn(dd[2], dd[2])) <=
                     r2;
            }
            near[hh] = nr;
            far[hh] = !nr;
        }
        const unsigned nm0 = __ballot_sync(FULL, near[0]), nm1 = __ballot_sync(FULL, near[1]);
        const unsigned fm0 = __ballot_sync(FULL, far[0]), fm1 = __ballot_sync(FULL, far[1]);
        int lpre = 0, lsum = 0;
        for (int w = 0; w < 8; ++w) {
            const int v = __shfl_sync(FULL, lc, w * 4);
            lpre += w < qw ? v : 0;
            lsum += v;
        }
        const int buf = it & 1;
        if (lane == 0) {
            s_w[buf][warp][0] = lsum;
            s_w[buf][warp][1] = __popc(fm0) + __popc(fm1);
            s_w[buf][warp][2] = __popc(nm0) + __popc(nm1);
        }
        __syncthreads();
        int oe = 0, of = 0, on = 0, te = 0, tf = 0, tn = 0;
        for (int w = 0; w < GW; ++w) {
            const int e0 = s_w[buf][w][0], f0 = s_w[buf][w][1], n0 = s_w[buf][w][2];
            if (w < warp) {
                oe += e0;
                of += f0;
                on += n0;
            }
            te += e0;
            tf += f0;
            tn += n0;
        }
        if (tail - head - nproc + tn > GLCAP) {   // the same in every thread
            if (tid == 0) atomicOr(err, ERR_GRAV_OVERFLOW);
            break;
        }
        if (FILL && leaf)
            for (int t = k; t < lc; t += 4) epj[be + ne + oe + lpre + t] = ci.z + t;
        // order within the warp: cell by cell, a cell's first children, then its second
        const int f_pre = __popc(fm0 & before) + __popc(fm1 & before), n_pre = __popc(nm0 & before) + __popc(nm1 & before);
        const int f_pos[2] = {f_pre + __popc(fm0 & cellm & below),
                              f_pre + __popc(fm0 & cellm) + __popc(fm1 & cellm & below)};
        const int n_pos[2] = {n_pre + __popc(nm0 & cellm & below),
                              n_pre + __popc(nm0 & cellm) + __popc(nm1 & cellm & below)};
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int ch = ci.x + k + 4 * hh;
            if (FILL && far[hh]) spj[bs + ns + of + f_pos[hh]] = ch;
            if (near[hh]) s_q[(tail + on + n_pos[hh]) & (GLCAP - 1)] = ch;
        }
        ne += te;
        ns += tf;
        head += nproc;
        tail += tn;
        __syncthreads();   // the queue entries written above
    }
    if (!FILL && tid == 0) {
        n_epj[g] = ne;
        n_spj[g] = ns;
    }
}

// the totals of the counting pass and its error word, for the host (pinned memory)
__global__ void k_list_totals(const int *oe, const int *ne, const int *os, const int *ns, const int *err, int *host) {
    after_previous();
    const int *p[5] = {oe, ne, os, ns, err};
    if (threadIdx.x == 0)
        for (int k = 0; k < 5; ++k) host[k] = *p[k];
}

}  // namespace sph

using namespace sph;

template <class T>
static int dalloc_l(sph_ctx *ctx, T **p, int64_t n) {
    if (*p) cudaFree(*p);
    *p = nullptr;
    if (n <= 0) n = 1;
    cudaError_t e = cudaMalloc((void **)p, sizeof(T) * (size_t)n);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return sph_fail(ctx, SPH_ERR_OOM, "device allocation of %lld bytes failed", (long long)(sizeof(T) * n));
    }
    return SPH_OK;
}

int sph_build_grav_lists(sph_ctx *ctx) {
    GravLists &G = ctx->grav;
    Tree &t = ctx->tree;
    cudaStream_t st = ctx->stream;
    const int ng = G.ng;
    int *hs = (int *)ctx->host_scalars;
    SPH_CUDA(ctx, cudaMemsetAsync(t.meta + META_ERR, 0, sizeof(int), st));
    k_grav_lists<false><<<ng, GL_T, 0, st>>>(
        ng, G.group_cell, FLD(ctx->F, SPH_X, ctx->cap), FLD(ctx->F, SPH_Y, ctx->cap), FLD(ctx->F, SPH_Z, ctx->cap),
        t.cinfo, t.level, t.com, t.rb, ctx->runs.prun, G.n_epj, G.n_spj, nullptr, nullptr, nullptr, nullptr,
        t.meta + META_ERR); ++ctx->launches;
    SPH_TRY(sph_scan_exclusive(ctx, G.n_epj, G.off_epj, nullptr, ng, nullptr));
    SPH_TRY(sph_scan_exclusive(ctx, G.n_spj, G.off_spj, nullptr, ng, nullptr));
    launch_after(true, k_list_totals, 1, 32, 0, st, G.off_epj + (ng - 1), G.n_epj + (ng - 1), G.off_spj + (ng - 1),
                 G.n_spj + (ng - 1), t.meta + META_ERR, hs); ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    SPH_CUDA(ctx, cudaStreamSynchronize(st));
    if (hs[4] & ERR_GRAV_OVERFLOW) return sph_fail(ctx, SPH_ERR_CAPACITY, "gravity walk stack overflow");
    const int64_t tot_e = (int64_t)hs[0] + hs[1], tot_s = (int64_t)hs[2] + hs[3];
    if (tot_e > 2000000000LL || tot_s > 2000000000LL)
        return sph_fail(ctx, SPH_ERR_CAPACITY, "gravity interaction lists exceed 2^31 entries");
    if (G.cap_epj < tot_e) {
        G.cap_epj = tot_e + tot_e / 4 + 1024;
        SPH_TRY(dalloc_l(ctx, &G.epj, G.cap_epj));
    }
    if (G.cap_spj < tot_s) {
        G.cap_spj = tot_s + tot_s / 4 + 1024;
        SPH_TRY(dalloc_l(ctx, &G.spj, G.cap_spj));
    }
    G.tot_epj = tot_e;
    G.tot_spj = tot_s;
    k_grav_lists<true><<<ng, GL_T, 0, st>>>(
        ng, G.group_cell, FLD(ctx->F, SPH_X, ctx->cap), FLD(ctx->F, SPH_Y, ctx->cap), FLD(ctx->F, SPH_Z, ctx->cap),
        t.cinfo, t.level, t.com, t.rb, ctx->runs.prun, G.n_epj, G.n_spj, G.off_epj, G.off_spj, G.epj, G.spj,
        t.meta + META_ERR); ++ctx->launches;
    SPH_CUDA(ctx, cudaGetLastError());
    G.valid = true;
    G.counts_valid = true;
    return SPH_OK;
}

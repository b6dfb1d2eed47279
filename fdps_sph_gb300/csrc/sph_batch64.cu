// FP64 functor kernels of the batch entry points: the reference functors (force.h:9-23, 89-106, 113-147,
// 154-168) on caller-supplied walks, in FP64.
//
// What bounds them is the FP64 pipe (sph_pair64.cuh), and 8 of 9 entries of an FDPS superset j-list lie
// outside the i-particle's support, where the density, derivative and hydro terms are exact zeros.  So a
// block takes IC i-particles of one walk, stages the walk's j entries tile by tile as FP32 positions relative
// to the walk's first i-particle, and each warp takes one i-particle at a time: its lanes test 32 j at a
// time in FP32 (about 20 instructions, off the FP64 pipe) with a bound on the rounding, the survivors queue
// up in shared memory, and every 32 of them are evaluated in FP64 from the payloads by a full warp.  A j that is
// dropped has a zero term for certain; everything the test cannot decide (NaN, infinities, non-positive
// smoothing lengths) is kept, so results are the functors' on any input.  The hydro functor's v_sig_max
// runs over the whole list: an out-of-support j is also kept unless FP32 with an error bound shows that
// another j's signal velocity is larger.  Partial sums meet by shuffles; the per-particle
// epilogues (divisions, the pow of the smoothing length) run once per block with one i-particle per lane.
//
// Against one thread per i-particle over the whole list in FP64, one 128-thread block per walk, a call of every
// functor: 180 particles in one walk 4,506 -> 152 us, 30,011 particles 63.7 -> 4.4 ms, staging, results and
// host included.
#include "sph_batch.cuh"
#include "sph_pair64.cuh"

namespace sph {

namespace {

constexpr int W = 8;            // most warps per block
constexpr int TJ = 512;         // j entries per tile
constexpr int IC_MAX = 32;      // i-particles per block
constexpr unsigned FULLW = 0xffffffffu;

__device__ __forceinline__ bool fin(double v) { return ((unsigned)__double2hiint(v) & 0x7ff00000u) != 0x7ff00000u; }

// FP32 bound on a coordinate's and a difference's rounding: 2^-21 of the 1-norms of both points
__device__ __forceinline__ float slack1(float x, float y, float z) {
    return 4.76837158203125e-07f * (fabsf(x) + fabsf(y) + fabsf(z));
}

// FP32 reach of a smoothing length: 2.5 h rounded up generously (2^-17), NaN (keeps everything) unless h is
// positive and finite
__device__ __forceinline__ float reach(double h) {
    const float H = (float)(SUPPORT * h) * 1.00000762939453125f;
    return (h > 0.0 && fin(h)) ? fmaxf(H, 1.0e-15f) : __int_as_float(0x7fffffff);
}

// one warp's queue of kept j entries: appended in list order, taken 32 at a time
struct Queue {
    int *buf;   // 64 entries of this warp
    int n;
    __device__ __forceinline__ void push(bool keep, int j, int lane) {
        const unsigned m = __ballot_sync(FULLW, keep);
        if (keep) buf[n + __popc(m & ((1u << lane) - 1u))] = j;
        n += __popc(m);
        __syncwarp();
    }
    // entry of this lane, -1 past the end; the first 32 leave the queue
    __device__ __forceinline__ int take(int lane) {
        const int j = lane < n ? buf[lane] : -1;
        const int rest = lane + 32 < n ? buf[lane + 32] : 0;
        __syncwarp();
        if (lane + 32 < n) buf[lane] = rest;
        n = n > 32 ? n - 32 : 0;
        __syncwarp();
        return j;
    }
};

// the walk's place in the staged arrays and this block's i-particles
struct Span {
    int64_t io, jo, nj, so, ns;
    int64_t i0;   // first i-particle of the block (within the walk)
    int ni;       // and how many
};

__device__ __forceinline__ Span span(const int64_t *meta, int64_t i0, int ic) {
    const int64_t *M = meta + 6 * blockIdx.x;
    Span s;
    s.io = M[0];
    s.jo = M[2];
    s.nj = M[3];
    s.so = M[4];
    s.ns = M[5];
    s.i0 = i0;
    s.ni = (int)min((int64_t)ic, M[1] - i0);
    return s;
}

// ---------------------------------------------------------------------------
// density

__global__ void __launch_bounds__(W * 32) k_walk_dens64(const int64_t *meta, int ic, const sph_epi_dens *epi,
                                                        JSrc<sph_epj_dens> epj, sph_result_dens *res) {
    __shared__ float4 s_j[TJ];          // x, y, z relative to the walk's first i-particle, slack
    __shared__ int s_q[W][64];
    __shared__ double s_i[IC_MAX][5];   // x, y, z, 1 / H (hi, lo)
    __shared__ float4 s_f[IC_MAX];      // the same in FP32: x, y, z, reach + slack
    __shared__ double s_sum[IC_MAX];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    for (int64_t i0 = (int64_t)blockIdx.y * ic; i0 < meta[6 * blockIdx.x + 1]; i0 += (int64_t)gridDim.y * ic) {
        const Span S = span(meta, i0, ic);
        __syncthreads();   // the last chunk's epilogue has read the shared sums
        const double cx = epi[S.io].pos[0], cy = epi[S.io].pos[1], cz = epi[S.io].pos[2];
        if (t < S.ni) {
            const sph_epi_dens &p = epi[S.io + S.i0 + t];
            s_i[t][0] = p.pos[0];
            s_i[t][1] = p.pos[1];
            s_i[t][2] = p.pos[2];
            const Inv64 iH = inv64(SUPPORT * p.smth);
            s_i[t][3] = iH.hi;
            s_i[t][4] = iH.lo;
            const float x = (float)(p.pos[0] - cx), y = (float)(p.pos[1] - cy), z = (float)(p.pos[2] - cz);
            s_f[t] = make_float4(x, y, z, reach(p.smth) + slack1(x, y, z));
            s_sum[t] = 0.0;
        }
        for (int64_t t0 = 0; t0 < S.nj; t0 += TJ) {
            const int tn = (int)min((int64_t)TJ, S.nj - t0);
            __syncthreads();
            for (int k = t; k < tn; k += blockDim.x) {
                const sph_epj_dens &q = epj[S.jo + t0 + k];
                const float x = (float)(q.pos[0] - cx), y = (float)(q.pos[1] - cy), z = (float)(q.pos[2] - cz);
                s_j[k] = make_float4(x, y, z, fin(q.mass) ? slack1(x, y, z) : __int_as_float(0x7fffffff));
            }
            __syncthreads();
            for (int i = warp; i < S.ni; i += nw) {
                const float4 f = s_f[i];
                const double xi = s_i[i][0], yi = s_i[i][1], zi = s_i[i][2];
                const Inv64 invH{s_i[i][3], s_i[i][4]};
                Queue Q{s_q[warp], 0};
                double sum = 0.0;
                auto eval = [&]() {
                    const int j = Q.take(lane);
                    if (j >= 0) {
                        const sph_epj_dens &q = epj[S.jo + t0 + j];
                        dens_pair64(q.pos[0] - xi, q.pos[1] - yi, q.pos[2] - zi, q.mass, invH, sum);
                    }
                };
                for (int k = lane; k < TJ && k - lane < tn; k += 32) {
                    bool keep = k < tn;
                    if (keep) {
                        const float4 p = s_j[k];
                        const float dx = p.x - f.x, dy = p.y - f.y, dz = p.z - f.z, rr = f.w + p.w;
                        keep = !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > rr * rr);   // false for NaN: kept
                    }
                    Q.push(keep, k, lane);
                    if (Q.n >= 32) eval();
                }
                if (Q.n > 0) eval();
                sum = warp_sum64(sum);
                if (lane == 0) s_sum[i] += sum;
            }
        }
        __syncthreads();
        if (t < S.ni) {
            const sph_epi_dens &p = epi[S.io + S.i0 + t];
            const double d = fmax(DENS_FLOOR, s_sum[t] * kernel_norm(SUPPORT * p.smth));
            sph_result_dens &o = res[S.io + S.i0 + t];
            o.dens = d;
            o.smth = SMTH_COEF * pow(p.mass / d, 1.0 / 3.0);
        }
    }
}

// ---------------------------------------------------------------------------
// derivative

__global__ void __launch_bounds__(W * 32) k_walk_drvt64(const int64_t *meta, int ic, const sph_epi_drvt *epi,
                                                        JSrc<sph_epj_drvt> epj, sph_result_drvt *res) {
    __shared__ float4 s_j[TJ];
    __shared__ int s_q[W][64];
    __shared__ double s_i[IC_MAX][10];   // x, v, 1 / H (hi, lo), H, 1e-6 h
    __shared__ float4 s_f[IC_MAX];
    __shared__ double s_sum[IC_MAX][6];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    for (int64_t i0 = (int64_t)blockIdx.y * ic; i0 < meta[6 * blockIdx.x + 1]; i0 += (int64_t)gridDim.y * ic) {
        const Span S = span(meta, i0, ic);
        __syncthreads();   // the last chunk's epilogue has read the shared sums
        const double cx = epi[S.io].pos[0], cy = epi[S.io].pos[1], cz = epi[S.io].pos[2];
        if (t < S.ni) {
            const sph_epi_drvt &p = epi[S.io + S.i0 + t];
            for (int d = 0; d < 3; ++d) {
                s_i[t][d] = p.pos[d];
                s_i[t][3 + d] = p.vel[d];
            }
            const Inv64 iH = inv64(SUPPORT * p.smth);
            s_i[t][6] = iH.hi;
            s_i[t][7] = iH.lo;
            s_i[t][8] = SUPPORT * p.smth;
            s_i[t][9] = 1.0e-6 * p.smth;
            const float x = (float)(p.pos[0] - cx), y = (float)(p.pos[1] - cy), z = (float)(p.pos[2] - cz);
            const bool ok = fin(p.vel[0]) && fin(p.vel[1]) && fin(p.vel[2]);
            s_f[t] = make_float4(x, y, z, ok ? reach(p.smth) + slack1(x, y, z) : __int_as_float(0x7fffffff));
            for (int d = 0; d < 6; ++d) s_sum[t][d] = 0.0;
        }
        for (int64_t t0 = 0; t0 < S.nj; t0 += TJ) {
            const int tn = (int)min((int64_t)TJ, S.nj - t0);
            __syncthreads();
            for (int k = t; k < tn; k += blockDim.x) {
                const sph_epj_drvt &q = epj[S.jo + t0 + k];
                const float x = (float)(q.pos[0] - cx), y = (float)(q.pos[1] - cy), z = (float)(q.pos[2] - cz);
                const bool ok = fin(q.mass) && fin(q.vel[0]) && fin(q.vel[1]) && fin(q.vel[2]);
                s_j[k] = make_float4(x, y, z, ok ? slack1(x, y, z) : __int_as_float(0x7fffffff));
            }
            __syncthreads();
            for (int i = warp; i < S.ni; i += nw) {
                const float4 f = s_f[i];
                const double *I = s_i[i];
                Queue Q{s_q[warp], 0};
                double D[6] = {0, 0, 0, 0, 0, 0};
                auto eval = [&]() {
                    const int j = Q.take(lane);
                    if (j >= 0) {
                        const sph_epj_drvt &q = epj[S.jo + t0 + j];
                        drvt_pair64(I[0] - q.pos[0], I[1] - q.pos[1], I[2] - q.pos[2], I[3] - q.vel[0], I[4] - q.vel[1],
                                    I[5] - q.vel[2], q.mass, Inv64{I[6], I[7]}, I[8], I[9], D);
                    }
                };
                for (int k = lane; k < TJ && k - lane < tn; k += 32) {
                    bool keep = k < tn;
                    if (keep) {
                        const float4 p = s_j[k];
                        const float dx = p.x - f.x, dy = p.y - f.y, dz = p.z - f.z, rr = f.w + p.w;
                        keep = !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > rr * rr);
                    }
                    Q.push(keep, k, lane);
                    if (Q.n >= 32) eval();
                }
                if (Q.n > 0) eval();
                const double s4 = warp_sum64x4(D), s5 = warp_sum64(D[4]), s6 = warp_sum64(D[5]);
                if ((lane & 7) == 0) s_sum[i][lane >> 3] += s4;
                if (lane == 0) {
                    s_sum[i][4] += s5;
                    s_sum[i][5] += s6;
                }
            }
        }
        __syncthreads();
        if (t < S.ni) {
            const sph_epi_drvt &p = epi[S.io + S.i0 + t];
            const double *D = s_sum[t];
            const double H = SUPPORT * p.smth, norm = kernel_norm(H), qn = -22.0 * norm / H;   // dW/dr / r per g
            const double gs = -(3.0 * norm * D[4] + qn * D[5]) / p.smth;
            const double c = -qn / p.dens;
            sph_result_drvt &o = res[S.io + S.i0 + t];
            o.grad_smth = 1.0 / (1.0 + p.smth * gs / (3.0 * p.dens));
            o.div_v = c * D[0];
            o.rot_v[0] = c * D[1];
            o.rot_v[1] = c * D[2];
            o.rot_v[2] = c * D[3];
        }
    }
}

// ---------------------------------------------------------------------------
// hydro

__device__ __forceinline__ Hydro64 hydro_of(const sph_epj_hydro &q) {
    return hydro64_consts(q.smth, q.dens, q.pres, q.grad_smth, q.Bal, q.snds);
}

__global__ void __launch_bounds__(W * 32) k_walk_hydro64(const int64_t *meta, int ic, const sph_epi_hydro *epi,
                                                         JSrc<sph_epj_hydro> epj, sph_result_hydro *res) {
    __shared__ float4 s_j[TJ];          // x, y, z, slack
    __shared__ float4 s_v[TJ];          // velocity relative to the walk's first i-particle, c_s
    __shared__ float s_h[TJ];           // reach of j
    __shared__ int s_q[W][64];
    __shared__ double s_i[IC_MAX][6];   // x, v
    __shared__ Hydro64 s_k[IC_MAX];
    __shared__ float4 s_f[IC_MAX], s_g[IC_MAX];   // x, y, z, reach; v, c_s
    __shared__ double s_sum[IC_MAX][5];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    for (int64_t i0 = (int64_t)blockIdx.y * ic; i0 < meta[6 * blockIdx.x + 1]; i0 += (int64_t)gridDim.y * ic) {
        const Span S = span(meta, i0, ic);
        __syncthreads();   // the last chunk's epilogue has read the shared sums
        const sph_epi_hydro &C = epi[S.io];
        const double cx = C.pos[0], cy = C.pos[1], cz = C.pos[2], ux = C.vel[0], uy = C.vel[1], uz = C.vel[2];
        if (t < S.ni) {
            const sph_epi_hydro &p = epi[S.io + S.i0 + t];
            bool ok = fin(p.dens) && fin(p.pres) && fin(p.snds) && fin(p.grad_smth) && fin(p.Bal) && p.dens > 0.0;
            for (int d = 0; d < 3; ++d) {
                s_i[t][d] = p.pos[d];
                s_i[t][3 + d] = p.vel[d];
                ok = ok && fin(p.vel[d]);
            }
            s_k[t] = hydro64_consts(p.smth, p.dens, p.pres, p.grad_smth, p.Bal, p.snds);
            const float x = (float)(p.pos[0] - cx), y = (float)(p.pos[1] - cy), z = (float)(p.pos[2] - cz);
            s_f[t] = make_float4(x, y, z, ok ? reach(p.smth) : __int_as_float(0x7fffffff));
            s_g[t] = make_float4((float)(p.vel[0] - ux), (float)(p.vel[1] - uy), (float)(p.vel[2] - uz), (float)p.snds);
            for (int d = 0; d < 5; ++d) s_sum[t][d] = 0.0;
        }
        for (int64_t t0 = 0; t0 < S.nj; t0 += TJ) {
            const int tn = (int)min((int64_t)TJ, S.nj - t0);
            __syncthreads();
            for (int k = t; k < tn; k += blockDim.x) {
                const sph_epj_hydro &q = epj[S.jo + t0 + k];
                const float x = (float)(q.pos[0] - cx), y = (float)(q.pos[1] - cy), z = (float)(q.pos[2] - cz);
                const bool ok = fin(q.mass) && fin(q.dens) && fin(q.pres) && fin(q.snds) && fin(q.grad_smth) &&
                                fin(q.Bal) && fin(q.vel[0]) && fin(q.vel[1]) && fin(q.vel[2]) && q.dens > 0.0;
                s_j[k] = make_float4(x, y, z, slack1(x, y, z));
                s_v[k] = make_float4((float)(q.vel[0] - ux), (float)(q.vel[1] - uy), (float)(q.vel[2] - uz),
                                     (float)q.snds);
                s_h[k] = ok ? reach(q.smth) : __int_as_float(0x7fffffff);
            }
            __syncthreads();
            for (int i = warp; i < S.ni; i += nw) {
                const float4 f = s_f[i], g = s_g[i];
                const float sl_i = slack1(f.x, f.y, f.z), ev_i = fabsf(g.x) + fabsf(g.y) + fabsf(g.z);
                const double *I = s_i[i];
                const Hydro64 K = s_k[i];
                Queue Q{s_q[warp], 0};
                double D[4] = {0, 0, 0, 0}, vmax = 0.0;
                float low = 0.0f;   // some j of this tile has a signal velocity of at least this (warp-uniform)
                auto eval = [&]() {
                    const int j = Q.take(lane);
                    if (j >= 0) {
                        const sph_epj_hydro &q = epj[S.jo + t0 + j];
                        hydro_pair64(I[0] - q.pos[0], I[1] - q.pos[1], I[2] - q.pos[2], I[3] - q.vel[0], I[4] - q.vel[1],
                                     I[5] - q.vel[2], q.mass, K, hydro_of(q), D, vmax);
                    }
                };
                for (int k = lane; k < TJ && k - lane < tn; k += 32) {
                    bool keep = false;
                    float vlo = 0.0f, vhi = 0.0f;
                    if (k < tn) {
                        const float4 p = s_j[k], v = s_v[k];
                        const float dx = f.x - p.x, dy = f.y - p.y, dz = f.z - p.z;
                        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                        const float sl = sl_i + p.w;
                        // the larger reach, a NaN of either winning (fmaxf would drop it)
                        const float hj = s_h[k], hm = f.w > hj ? f.w : (f.w <= hj ? hj : __int_as_float(0x7fffffff));
                        const float rr = hm + sl;
                        // inside, undecidable, or too close to a rounding of the position for the bound on v_sig below
                        keep = !(r2 > rr * rr) || !(sl * sl < 2.3283064365386963e-10f * r2) || !(r2 < 1.0e37f);   // 2^-32
                        const float wx = g.x - v.x, wy = g.y - v.y, wz = g.z - v.z;
                        const float w = fminf(fmaf(wx, dx, fmaf(wy, dy, wz * dz)), 0.0f) * rsqrt_a(r2);
                        const float cs = g.w + v.w, vs = fmaf(-3.0f, w, cs);
                        const float ev = ev_i + fabsf(v.x) + fabsf(v.y) + fabsf(v.z);
                        const float err = 6.103515625e-05f * (fabsf(g.w) + fabsf(v.w) + 3.0f * ev);   // 2^-14
                        keep = keep || !(err < 1.0e15f);   // (no product above overflows below that)
                        vlo = keep ? 0.0f : fmaxf(vs - err, 0.0f);
                        vhi = vs + err;
                    }
                    low = fmaxf(low, __int_as_float(__reduce_max_sync(FULLW, __float_as_int(vlo))));
                    if (k < tn && !keep) keep = !(vhi < low);
                    Q.push(keep, k, lane);
                    if (Q.n >= 32) eval();
                }
                if (Q.n > 0) eval();
                const double s4 = warp_sum64x4(D);
    #pragma unroll
                for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_xor_sync(FULLW, vmax, o));
                if ((lane & 7) == 0) s_sum[i][lane >> 3] += s4;
                if (lane == 0) s_sum[i][4] = fmax(s_sum[i][4], vmax);
            }
        }
        __syncthreads();
        if (t < S.ni) {
            const double *D = s_sum[t];
            sph_result_hydro &o = res[S.io + S.i0 + t];
            o.acc[0] = D[0];
            o.acc[1] = D[1];
            o.acc[2] = D[2];
            o.eng_dot = 0.5 * D[3];
            o.dt = C_CFL * 2.0 * epi[S.io + S.i0 + t].smth / D[4];
        }
    }
}

// ---------------------------------------------------------------------------
// gravity: every j counts, so the lanes split the list, 32 j of an i-particle at a time

__global__ void __launch_bounds__(W * 32) k_walk_grav64(const int64_t *meta, int ic, const sph_epi_grav *epi,
                                                        JSrc<sph_epj_grav> epj, JSrc<sph_spj_monopole> spj,
                                                        sph_result_grav *res) {
    constexpr int TG = 512;
    __shared__ double s_x[4][TG];   // x, y, z, G m
    __shared__ double s_i[IC_MAX][4];
    __shared__ double s_sum[IC_MAX][4];
    const double G = 6.67e-11;   // force.h:171-172
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    for (int64_t i0 = (int64_t)blockIdx.y * ic; i0 < meta[6 * blockIdx.x + 1]; i0 += (int64_t)gridDim.y * ic) {
        const Span S = span(meta, i0, ic);
        __syncthreads();   // the last chunk's epilogue has read the shared sums
        if (t < S.ni) {
            const sph_epi_grav &p = epi[S.io + S.i0 + t];
            for (int d = 0; d < 3; ++d) s_i[t][d] = p.pos[d];
            s_i[t][3] = p.eps2;
            for (int d = 0; d < 4; ++d) s_sum[t][d] = 0.0;
        }
        const int64_t nl = S.nj + S.ns;   // EPJ, then SPJ
        for (int64_t t0 = 0; t0 < nl; t0 += TG) {
            const int tn = (int)min((int64_t)TG, nl - t0);
            __syncthreads();
            for (int k = t; k < tn; k += blockDim.x) {
                const int64_t e = t0 + k;
                const double *pos;
                double m;
                if (e < S.nj) {
                    const sph_epj_grav &q = epj[S.jo + e];
                    pos = q.pos;
                    m = q.mass;
                } else {
                    const sph_spj_monopole &q = spj[S.so + e - S.nj];
                    pos = q.pos;
                    m = q.mass;
                }
                for (int d = 0; d < 3; ++d) s_x[d][k] = pos[d];
                s_x[3][k] = G * m;
            }
            __syncthreads();
            for (int i = warp; i < S.ni; i += nw) {
                const double xi = s_i[i][0], yi = s_i[i][1], zi = s_i[i][2], e2 = s_i[i][3];
                double A[4] = {0, 0, 0, 0};
    #pragma unroll 2
                for (int k = lane; k < tn; k += 32)
                    grav_pair64(xi - s_x[0][k], yi - s_x[1][k], zi - s_x[2][k], e2, s_x[3][k], A);
                const double s4 = warp_sum64x4(A);
                if ((lane & 7) == 0) s_sum[i][lane >> 3] += s4;
            }
        }
        __syncthreads();
        if (t < S.ni) {
            const double *A = s_sum[t];
            sph_result_grav &o = res[S.io + S.i0 + t];
            o.acc[0] = A[0];
            o.acc[1] = A[1];
            o.acc[2] = A[2];
            o.pot = A[3];
            o.dt = 1.0e30;   // RESULT::Grav::clear(), dt untouched by the functor
        }
    }
}

// Blocks of 8 warps with 32 i-particles (four per warp, one staging of the j-list for them) where that still
// gives every SM two blocks, else with 8 (one per warp), so that a few walks spread over the chip, and for
// the smallest dispatches 4 warps with one i-particle each, so that every warp has an FP64 pipe (one per SM quarter)
// to itself: a call of every functor on one walk of 180 particles 168 -> 152 us.
struct Shape {
    int ic, threads;
    dim3 grid;
    Shape(int n_walk, int64_t n_i, int max_i) {
        ic = n_i >= GB300_SMS * 64 ? IC_MAX : (n_i > GB300_SMS * 4 ? W : 4);
        threads = ic == 4 ? 128 : W * 32;
        const int chunks = (max_i + ic - 1) / ic;
        grid = dim3((unsigned)n_walk, (unsigned)(chunks > 0 ? (chunks < 4096 ? chunks : 4096) : 1));
    }
};

}  // namespace

void batch64_dens(int n_walk, int64_t n_i, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_dens *epi,
                  JSrc<sph_epj_dens> epj, sph_result_dens *res) {
    const Shape s(n_walk, n_i, max_i);
    k_walk_dens64<<<s.grid, s.threads, 0, st>>>(meta, s.ic, epi, epj, res);
}
void batch64_drvt(int n_walk, int64_t n_i, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_drvt *epi,
                  JSrc<sph_epj_drvt> epj, sph_result_drvt *res) {
    const Shape s(n_walk, n_i, max_i);
    k_walk_drvt64<<<s.grid, s.threads, 0, st>>>(meta, s.ic, epi, epj, res);
}
void batch64_hydro(int n_walk, int64_t n_i, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_hydro *epi,
                   JSrc<sph_epj_hydro> epj, sph_result_hydro *res) {
    const Shape s(n_walk, n_i, max_i);
    k_walk_hydro64<<<s.grid, s.threads, 0, st>>>(meta, s.ic, epi, epj, res);
}
void batch64_grav(int n_walk, int64_t n_i, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_grav *epi,
                  JSrc<sph_epj_grav> epj, JSrc<sph_spj_monopole> spj, sph_result_grav *res) {
    const Shape s(n_walk, n_i, max_i);
    k_walk_grav64<<<s.grid, s.threads, 0, st>>>(meta, s.ic, epi, epj, spj, res);
}

}  // namespace sph

// Mixed-precision functor kernels for the batch entry points (sph_dispatch_* after
// sph_batch_set_precision(SPH_PREC_MIXED)).
//
// The same walks and results as the FP64 kernels of sph_batch64.cu (the reference functors,
// force.h:9-23, 89-106, 113-147, 154-168), with the pair arithmetic of the device-resident mixed
// path: positions and velocities relative to the walk's first i-particle as double-floats (hi + lo
// FP32 pairs formed from the FP64 payload once per particle), pair terms in FP32 with the
// approximate root / reciprocal instructions, masses in units of one mass of the walk and the
// kernel normalisation of the i-particle factored out of the sums, FP32 partial sums of 32 terms
// added into compensated FP32 accumulators, and the per-particle epilogue (density floor and h, grad-h
// factor, dt, the normalisation) in FP64.
#include "sph_batch.cuh"

using namespace sph;

namespace {

// A block takes the walk's i-particles 32 at a time, four lanes per i-particle, and the j-list (gravity: EPJ, then SPJ) in
// tiles of 128 entries.  The sums' order is that of one thread over the list: FP32 partial sums of 32 consecutive
// entries, added block by block into the compensated pair.  Lane q sums the tile's q-th block of 32, then the lanes
// exchange their partial sums so that lane q adds component q of all four in block order: the bits are one thread's.
// One thread per i-particle in a block per walk had five warps on an SM (a dispatch of 256 walks, 93 i-particles each),
// bound by latency, read each j as scalars and did the FP64 preparation of every i-particle in idle lanes too.
//
// A dispatch alone is bound by the latency of its tiles (staging, barriers, a serial chain of 32 terms a lane).  Where the
// dispatches of several tags follow each other it is the gather of the next walks over the host link, and what counts is
// that its blocks find room beside these: with 64 registers a thread a dispatch of 256 walks and the end of the one
// before fill the register file, and the gather waits.  So the lanes keep one component each instead of four (which also
// takes two thirds of the exchange), walk sizes are 32-bit, and registers are held to 48 (56 for the derivative; the
// compiler puts part of the preparation on the stack).  Density / derivative / hydro / gravity, us a dispatch of 256
// walks in payload form, host link and calls included, four tags in turn:
//                                           100,000 particles (93 i a walk)   1M (84 i, 800 to 2,200 j)
//   thread per i, one block per walk            93 / 168 / 230 / 157              86 / 138 / 194 / 155
//   four lanes, 64 registers                    76 / 115 / 176 / 132              92 / 137 / 214 / 185
//   with one component a lane                   77 / 109 / 170 / 122              92 / 134 / 209 / 176
//   and 48 to 56 registers                      75 / 106 / 173 / 117              84 / 125 / 186 / 151
// and one walk after the other, 4,000 particles (66 walks, a dispatch): 66 / 107 / 147 / 102 -> 66 / 97 / 144 / 84.  A pass
// of every functor, index form: 100,003 particles 3.06 (thread per i) -> 2.12 -> 1.95 ms, 1M 23.1 -> 19.7 -> 17.2 ms;
// payload form, 1M: 28.1 -> 31.4 -> 26.9 ms.  40 registers: hydro of 1M 212.  Two lanes per i-particle (64 i a block)
// leave more room still (1M payload 25.5 ms) but are 7 to 14% slower from 1,500 to 30,000 particles; blocks of 256 and
// 384 threads, 64 threads, and one lane are slower than both.
constexpr int LQ = 4;                  // lanes per i-particle
constexpr int BT = 128;                // threads per block
constexpr int BI = BT / LQ;            // i-particles per block
constexpr int TJ = 32 * LQ;            // entries per tile
constexpr int TP = 33 * LQ;            // its shared-memory slots: a slot of padding per 32 entries, so that the four
                                       // lanes' float4 reads fall into different banks
__device__ __forceinline__ int slot(int t) { return t + (t >> 5); }

__device__ __forceinline__ float4 hi4(const double *p, const double3 o, float w, float4 *lo, float lw) {
    float a, b, c, d, e, f;
    split_df(p[0] - o.x, a, d);
    split_df(p[1] - o.y, b, e);
    split_df(p[2] - o.z, c, f);
    *lo = make_float4(d, e, f, lw);
    return make_float4(a, b, c, w);
}

// m / m0, without the division (7.5 FP64 instructions) for the equal masses of most runs
__device__ __forceinline__ float in_units(double m, double m0) {
    return __double_as_longlong(m) == __double_as_longlong(m0) ? 1.0f : (float)(m / m0);
}

__device__ __forceinline__ float dfd(float ah, float al, float bh, float bl) { return (ah - bh) + (al - bl); }

// The compensated sums of one i-particle's Q components.  Of four and more, lane q keeps component q; the fifth, or the
// only one, is kept by every lane.
template <int Q>
struct Sums {
    static constexpr int A = Q >= LQ ? LQ : 0, R = Q - A;   // components kept by one lane each, by all
    float P[Q];                                             // this lane's block
    float Dh = 0.0f, Dl = 0.0f, rest = 0.0f;                // compensated sum, the list's last, partial block
    float Eh[R + 1], El[R + 1], rest_all[R + 1];
    __device__ __forceinline__ Sums() {
#pragma unroll
        for (int q = 0; q < Q; ++q) P[q] = 0.0f;
#pragma unroll
        for (int q = 0; q < R; ++q) Eh[q] = El[q] = rest_all[q] = 0.0f;
    }
    // the lanes' blocks b0 .. b0 + 3 of a list with n_full whole blocks, in order
    __device__ __forceinline__ void add(unsigned b0, unsigned n_full) {
        const unsigned mask = 0xfu << (threadIdx.x & 28);
        if constexpr (A > 0) {
            const bool odd = threadIdx.x & 1, high = threadIdx.x & 2;
            // v[l] becomes lane l's partial sum of this lane's component (a 4 x 4 transpose)
            float v[LQ];
#pragma unroll
            for (int l = 0; l < LQ; ++l) v[l] = P[l];
            float s0 = __shfl_xor_sync(mask, odd ? v[0] : v[1], 1), s1 = __shfl_xor_sync(mask, odd ? v[2] : v[3], 1);
            v[0] = odd ? s0 : v[0];
            v[1] = odd ? v[1] : s0;
            v[2] = odd ? s1 : v[2];
            v[3] = odd ? v[3] : s1;
            s0 = __shfl_xor_sync(mask, high ? v[0] : v[2], 2);
            s1 = __shfl_xor_sync(mask, high ? v[1] : v[3], 2);
            v[0] = high ? s0 : v[0];
            v[1] = high ? s1 : v[1];
            v[2] = high ? v[2] : s0;
            v[3] = high ? v[3] : s1;
#pragma unroll
            for (int l = 0; l < LQ; ++l) {
                if (b0 + l < n_full) df_add(Dh, Dl, v[l]);
                else if (b0 + l == n_full) rest = v[l];
            }
        }
#pragma unroll
        for (int l = 0; l < LQ; ++l)
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const float v = __shfl_sync(mask, P[A + q], l, LQ);
                if (b0 + l < n_full) df_add(Eh[q], El[q], v);
                else if (b0 + l == n_full) rest_all[q] = v;
            }
#pragma unroll
        for (int q = 0; q < Q; ++q) P[q] = 0.0f;
    }
    // the sums of this i-particle to shared memory
    __device__ __forceinline__ void store(float2 *out) {
        if constexpr (A > 0) {
            df_add(Dh, Dl, rest);
            out[threadIdx.x % LQ] = make_float2(Dh, Dl);
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
            df_add(Eh[q], El[q], rest_all[q]);
            if (threadIdx.x % LQ == 0) out[A + q] = make_float2(Eh[q], El[q]);
        }
    }
};

__device__ __forceinline__ double total(float2 d) { return (double)d.x + (double)d.y; }

// the block's walk and the loop over its i-particles
struct Walk {
    int64_t io, jo, so;
    unsigned ni, nj, ns;   // (n_epi, n_epj, n_spj of the call: below 2^31, a sum of two below 2^32)
    unsigned sub;          // lane of the i-particle
    __device__ __forceinline__ explicit Walk(const int64_t *meta) {
        const int64_t *M = meta + 6 * blockIdx.x;
        io = M[0];
        ni = (unsigned)M[1];
        jo = M[2];
        nj = (unsigned)M[3];
        so = M[4];
        ns = (unsigned)M[5];
        sub = threadIdx.x % LQ;
    }
    // entries of this lane's block of a tile of tn entries
    __device__ __forceinline__ int count(unsigned tn) const { return max(0, min(32, (int)tn - 32 * (int)sub)); }
};

// CalcDensity: rho = max(5, norm sum m_j W), h = 1.2 (m / rho)^(1/3)
__global__ void __launch_bounds__(BT, 10) k_walk_dens32(const int64_t *meta, const sph_epi_dens *epi,
                                                     JSrc<sph_epj_dens> epj, sph_result_dens *res) {
    __shared__ float4 sp[TP], sl[TP];   // position hi, mass; lo
    __shared__ float4 ip[BI], il[BI];   // of the i-particles: position hi, 1 / H; lo
    __shared__ float2 is[BI];
    const Walk W(meta);
    if (W.ni == 0) return;
    const double3 o = make_double3(epi[W.io].pos[0], epi[W.io].pos[1], epi[W.io].pos[2]);
    const double m0 = epi[W.io].mass > 0.0 ? epi[W.io].mass : 1.0;   // the walk's mass unit (FP32 range)
    for (unsigned i0 = blockIdx.y * BI; i0 < W.ni; i0 += gridDim.y * BI) {
        const unsigned g = threadIdx.x / LQ;   // this lane's i-particle of the block's
        const bool act = i0 + g < W.ni;
        const unsigned im = i0 + threadIdx.x;   // the i-particle this thread prepares and finishes
        const bool mine = threadIdx.x < BI && im < W.ni;
        const unsigned s0 = 33 * W.sub;   // the first slot of this lane's block
        if (mine) {
            const sph_epi_dens &I = epi[W.io + im];
            ip[threadIdx.x] = hi4(I.pos, o, (float)(1.0 / (SUPPORT * I.smth)), &il[threadIdx.x], 0.0f);
        }
        __syncthreads();
        const float4 ph = ip[g], pl = il[g];
        const float invH = ph.w;
        Sums<1> S;
        for (unsigned tile = 0; tile < (W.nj + (TJ - 1ull)) / TJ; ++tile) {
            const unsigned t0 = tile * TJ, tn = min((unsigned)TJ, W.nj - t0);
            for (unsigned k = threadIdx.x; k < tn; k += BT) {
                const sph_epj_dens &q = epj[W.jo + t0 + k];
                sp[slot(k)] = hi4(q.pos, o, in_units(q.mass, m0), &sl[slot(k)], 0.0f);
            }
            __syncthreads();
            const int tc = act ? W.count(tn) : 0;
#pragma unroll 2
            for (int t = 0; t < tc; ++t) {
                const float4 qh = sp[s0 + t], ql = sl[s0 + t];
                const float dx = dfd(qh.x, ql.x, ph.x, pl.x), dy = dfd(qh.y, ql.y, ph.y, pl.y),
                            dz = dfd(qh.z, ql.z, ph.z, pl.z);
                const float s = sqrt_a(dx * dx + dy * dy + dz * dz) * invH;
                const float p = fmaxf(1.0f - s, 0.0f), p2 = p * p, p4 = p2 * p2;
                S.P[0] = fmaf(qh.w, (1.0f + s * (8.0f + s * (25.0f + s * 32.0f))) * (p4 * p4), S.P[0]);
            }
            if (act) S.add(4 * tile, W.nj / 32);
            __syncthreads();
        }
        S.store(&is[g]);
        __syncthreads();
        if (mine) {
            const sph_epi_dens &I = epi[W.io + im];
            const double d = fmax(DENS_FLOOR, total(is[threadIdx.x]) * m0 * kernel_norm(SUPPORT * I.smth));
            res[W.io + im].dens = d;
            res[W.io + im].smth = SMTH_COEF * cbrt(I.mass / d);
        }
        __syncthreads();
    }
}

// CalcDerivative + grad-h factor: div v, rot v, grad_smth (force.h:89-106)
__global__ void __launch_bounds__(BT, 9) k_walk_drvt32(const int64_t *meta, const sph_epi_drvt *epi,
                                                     JSrc<sph_epj_drvt> epj, sph_result_drvt *res) {
    __shared__ float4 sp[TP], sl[TP], sv[TP], su[TP];   // position hi, mass; lo; velocity hi; lo
    // of the i-particles: position hi, 1 / H; lo, H; velocity hi, 1e-6 h; lo
    __shared__ float4 ip[BI], il[BI], iv[BI], iu[BI];
    __shared__ float2 is[BI][5];
    const Walk W(meta);
    if (W.ni == 0) return;
    const double3 o = make_double3(epi[W.io].pos[0], epi[W.io].pos[1], epi[W.io].pos[2]);
    const double3 ov = make_double3(epi[W.io].vel[0], epi[W.io].vel[1], epi[W.io].vel[2]);
    const double m0 = (W.nj > 0 && epj[W.jo].mass > 0.0) ? epj[W.jo].mass : 1.0;   // the walk's mass unit
    for (unsigned i0 = blockIdx.y * BI; i0 < W.ni; i0 += gridDim.y * BI) {
        const unsigned g = threadIdx.x / LQ;   // this lane's i-particle of the block's
        const bool act = i0 + g < W.ni;
        const unsigned im = i0 + threadIdx.x;   // the i-particle this thread prepares and finishes
        const bool mine = threadIdx.x < BI && im < W.ni;
        const unsigned s0 = 33 * W.sub;   // the first slot of this lane's block
        if (mine) {
            const sph_epi_drvt &I = epi[W.io + im];
            const double H = SUPPORT * I.smth;
            ip[threadIdx.x] = hi4(I.pos, o, (float)(1.0 / H), &il[threadIdx.x], (float)H);
            iv[threadIdx.x] = hi4(I.vel, ov, (float)(1.0e-6 * I.smth), &iu[threadIdx.x], 0.0f);
        }
        __syncthreads();
        const float4 ph = ip[g], pl = il[g], vh = iv[g], vl = iu[g];
        const float invH = ph.w, Hf = pl.w, ceps = vh.w;
        Sums<5> S;
        for (unsigned tile = 0; tile < (W.nj + (TJ - 1ull)) / TJ; ++tile) {
            const unsigned t0 = tile * TJ, tn = min((unsigned)TJ, W.nj - t0);
            for (unsigned k = threadIdx.x; k < tn; k += BT) {
                const sph_epj_drvt &q = epj[W.jo + t0 + k];
                sp[slot(k)] = hi4(q.pos, o, in_units(q.mass, m0), &sl[slot(k)], 0.0f);
                sv[slot(k)] = hi4(q.vel, ov, 0.0f, &su[slot(k)], 0.0f);
            }
            __syncthreads();
            const int tc = act ? W.count(tn) : 0;
#pragma unroll 1
            for (int t = 0; t < tc; ++t) {
                const float4 qh = sp[s0 + t], ql = sl[s0 + t], uh = sv[s0 + t], ul = su[s0 + t];
                const float dx = dfd(ph.x, pl.x, qh.x, ql.x), dy = dfd(ph.y, pl.y, qh.y, ql.y),
                            dz = dfd(ph.z, pl.z, qh.z, ql.z);
                const float wx = dfd(uh.x, ul.x, vh.x, vl.x), wy = dfd(uh.y, ul.y, vh.y, vl.y),
                            wz = dfd(uh.z, ul.z, vh.z, vl.z);   // v_j - v_i
                const float rr2 = dx * dx + dy * dy + dz * dz;
                const float r = sqrt_a(rr2);
                float w, g;
                wendland_poly_f(r * invH, w, g);
                const float gf = g * rcp_a(r * Hf + ceps);
                const float m = qh.w;
                S.P[0] = fmaf(m * gf, wx * dx + wy * dy + wz * dz, S.P[0]);
                S.P[1] = fmaf(m * gf, wy * dz - wz * dy, S.P[1]);
                S.P[2] = fmaf(m * gf, wz * dx - wx * dz, S.P[2]);
                S.P[3] = fmaf(m * gf, wx * dy - wy * dx, S.P[3]);
                S.P[4] = fmaf(m, 3.0f * w + gf * rr2, S.P[4]);
            }
            if (act) S.add(4 * tile, W.nj / 32);
            __syncthreads();
        }
        S.store(is[g]);
        __syncthreads();
        if (mine) {
            const sph_epi_drvt &I = epi[W.io + im];
            const double hi = I.smth, rhoi = I.dens, norm = m0 * kernel_norm(SUPPORT * hi);
            double D[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) D[k] = total(is[threadIdx.x][k]) * norm;
            const double gs = -D[4] / hi;
            sph_result_drvt &out = res[W.io + im];
            out.grad_smth = 1.0 / (1.0 + hi * gs / (3.0 * rhoi));
            out.div_v = D[0] / rhoi;
            out.rot_v[0] = D[1] / rhoi;
            out.rot_v[1] = D[2] / rhoi;
            out.rot_v[2] = D[3] / rhoi;
        }
        __syncthreads();
    }
}

// CalcHydroForce: acceleration, du/dt, dt (force.h:113-147)
__global__ void __launch_bounds__(BT, 10) k_walk_hydro32(const int64_t *meta, const sph_epi_hydro *epi,
                                                      JSrc<sph_epj_hydro> epj, sph_result_hydro *res) {
    // position hi, mass; lo, H; velocity hi, 1 / H; lo, rho; f P / rho^2, c_s, f, Bal
    __shared__ float4 sp[TP], sl[TP], sv[TP], su[TP], sa[TP];
    // of the i-particles: position hi, 1 / H; lo, H; velocity hi, 1e-6 h; lo, rho; f P / rho^2, c_s, f, Bal
    __shared__ float4 ip[BI], il[BI], iv[BI], iu[BI], ia[BI];
    __shared__ float2 is[BI][4];
    __shared__ float iw[BI];   // v_sig_max
    const Walk W(meta);
    if (W.ni == 0) return;
    const double3 o = make_double3(epi[W.io].pos[0], epi[W.io].pos[1], epi[W.io].pos[2]);
    const double3 ov = make_double3(epi[W.io].vel[0], epi[W.io].vel[1], epi[W.io].vel[2]);
    const double m0 = (W.nj > 0 && epj[W.jo].mass > 0.0) ? epj[W.jo].mass : 1.0;   // the walk's mass unit
    for (unsigned i0 = blockIdx.y * BI; i0 < W.ni; i0 += gridDim.y * BI) {
        const unsigned g = threadIdx.x / LQ;   // this lane's i-particle of the block's
        const bool act = i0 + g < W.ni;
        const unsigned im = i0 + threadIdx.x;   // the i-particle this thread prepares and finishes
        const bool mine = threadIdx.x < BI && im < W.ni;
        const unsigned s0 = 33 * W.sub;   // the first slot of this lane's block
        if (mine) {
            const sph_epi_hydro &I = epi[W.io + im];
            const double H = SUPPORT * I.smth;
            ip[threadIdx.x] = hi4(I.pos, o, (float)(1.0 / H), &il[threadIdx.x], (float)H);
            iv[threadIdx.x] = hi4(I.vel, ov, (float)(1.0e-6 * I.smth), &iu[threadIdx.x], (float)I.dens);
            ia[threadIdx.x] = make_float4((float)(I.grad_smth * I.pres / (I.dens * I.dens)), (float)I.snds,
                                          (float)I.grad_smth, (float)I.Bal);
        }
        __syncthreads();
        const float4 ph = ip[g], pl = il[g], vh = iv[g], vl = iu[g], I4 = ia[g];
        const float invHi = ph.w, Hi = pl.w, cepsi = vh.w, rhof = vl.w, Ai = I4.x, cf = I4.y, ff = I4.z, bf = I4.w;
        Sums<4> S;
        float vmax = 0.0f;
        for (unsigned tile = 0; tile < (W.nj + (TJ - 1ull)) / TJ; ++tile) {
            const unsigned t0 = tile * TJ, tn = min((unsigned)TJ, W.nj - t0);
            for (unsigned k = threadIdx.x; k < tn; k += BT) {
                const sph_epj_hydro &q = epj[W.jo + t0 + k];
                const double Hj = SUPPORT * q.smth;
                sp[slot(k)] = hi4(q.pos, o, in_units(q.mass, m0), &sl[slot(k)], (float)Hj);
                sv[slot(k)] = hi4(q.vel, ov, (float)(1.0 / Hj), &su[slot(k)], (float)q.dens);
                sa[slot(k)] = make_float4((float)(q.grad_smth * q.pres / (q.dens * q.dens)), (float)q.snds,
                                          (float)q.grad_smth, (float)q.Bal);
            }
            __syncthreads();
            const int tc = act ? W.count(tn) : 0;
#pragma unroll 1
            for (int t = 0; t < tc; ++t) {
                const float4 qh = sp[s0 + t], ql = sl[s0 + t], uh = sv[s0 + t], ul = su[s0 + t], J = sa[s0 + t];
                const float jH = ql.w, jinvH = uh.w;
                const float dx = dfd(ph.x, pl.x, qh.x, ql.x), dy = dfd(ph.y, pl.y, qh.y, ql.y),
                            dz = dfd(ph.z, pl.z, qh.z, ql.z);
                const float wx = dfd(vh.x, vl.x, uh.x, ul.x), wy = dfd(vh.y, vl.y, uh.y, ul.y),
                            wz = dfd(vh.z, vl.z, uh.z, ul.z);
                const float rr2 = dx * dx + dy * dy + dz * dz;
                const float r = sqrt_a(rr2);
                const float dvdr = wx * dx + wy * dy + wz * dz;
                const float w = (dvdr < 0.0f) ? dvdr * rcp_a(r) : 0.0f;
                const float vsig = cf + J.y - 3.0f * w;
                vmax = fmaxf(vmax, vsig);
                const float AV = -0.5f * vsig * w * rcp_a(0.5f * (rhof + ul.w)) * 0.5f * (bf + J.w);
                float wi_, gi_, wj_, gj_;
                wendland_poly_f(r * invHi, wi_, gi_);
                wendland_poly_f(r * jinvH, wj_, gj_);
                const float nr = Hi * jinvH;   // the j kernel's normalisation relative to the i kernel's
                const float gfi = gi_ * rcp_a(r * Hi + cepsi);
                const float gfj = (nr * nr * nr) * gj_ * rcp_a(fmaf(r, jH, 4.0e-7f * jH));
                const float gws = 0.5f * (gfi * ff + gfj * J.z);
                const float coef = qh.w * (Ai * gfi + J.x * gfj + AV * gws);
                S.P[0] = fmaf(-coef, dx, S.P[0]);
                S.P[1] = fmaf(-coef, dy, S.P[1]);
                S.P[2] = fmaf(-coef, dz, S.P[2]);
                S.P[3] = fmaf(qh.w * (Ai + 0.5f * AV) * gws, dvdr, S.P[3]);
            }
            if (act) S.add(4 * tile, W.nj / 32);
            __syncthreads();
        }
        const unsigned mask = 0xfu << (threadIdx.x & 28);
        for (int off = LQ / 2; off > 0; off >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(mask, vmax, off, LQ));
        S.store(is[g]);
        if (W.sub == 0) iw[g] = vmax;
        __syncthreads();
        if (mine) {
            const double hi = epi[W.io + im].smth, norm = m0 * kernel_norm(SUPPORT * hi);
            double D[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) D[k] = total(is[threadIdx.x][k]) * norm;
            sph_result_hydro &out = res[W.io + im];
            out.acc[0] = D[0];
            out.acc[1] = D[1];
            out.acc[2] = D[2];
            out.eng_dot = D[3];
            out.dt = C_CFL * 2.0 * hi / (double)iw[threadIdx.x];
        }
        __syncthreads();
    }
}

// CalcGravityForce<EPJ::Grav> then <SPJMonopole> (force.h:154-168): G m folded into the tile
__global__ void __launch_bounds__(BT, 10) k_walk_grav32(const int64_t *meta, const sph_epi_grav *epi,
                                                     JSrc<sph_epj_grav> epj, JSrc<sph_spj_monopole> spj,
                                                     sph_result_grav *res) {
    __shared__ float4 sp[TP], sl[TP];   // position hi, G m; lo
    __shared__ float4 ip[BI], il[BI];   // of the i-particles: position hi, eps^2; lo
    __shared__ float2 is[BI][4];
    const double G = 6.67e-11;   // force.h:171-172
    const Walk W(meta);
    if (W.ni == 0) return;
    const double3 o = make_double3(epi[W.io].pos[0], epi[W.io].pos[1], epi[W.io].pos[2]);
    // G m in units of the walk's first EPJ mass (or SPJ mass) keeps the FP32 products in range; a mass that is no unit
    // (0 x G m / 0 would be a NaN in every sum of the walk) leaves them as they are
    const double m0 = W.nj > 0 ? epj[W.jo].mass : (W.ns > 0 ? spj[W.so].mass : 1.0);
    const double gscale = G * (m0 != 0.0 && isfinite(m0) ? m0 : 1.0);
    const unsigned nl = W.nj + W.ns;
    for (unsigned i0 = blockIdx.y * BI; i0 < W.ni; i0 += gridDim.y * BI) {
        const unsigned g = threadIdx.x / LQ;   // this lane's i-particle of the block's
        const bool act = i0 + g < W.ni;
        const unsigned im = i0 + threadIdx.x;   // the i-particle this thread prepares and finishes
        const bool mine = threadIdx.x < BI && im < W.ni;
        const unsigned s0 = 33 * W.sub;   // the first slot of this lane's block
        if (mine)
            ip[threadIdx.x] = hi4(epi[W.io + im].pos, o, (float)epi[W.io + im].eps2, &il[threadIdx.x], 0.0f);
        __syncthreads();
        const float4 ph = ip[g], pl = il[g];
        const float e2 = ph.w;
        Sums<4> S;
        for (unsigned tile = 0; tile < (nl + (TJ - 1ull)) / TJ; ++tile) {
            const unsigned t0 = tile * TJ, tn = min((unsigned)TJ, nl - t0);
            for (unsigned k = threadIdx.x; k < tn; k += BT) {
                const unsigned e = t0 + k;
                const double *pp;
                double mm;
                if (e < W.nj) {
                    const sph_epj_grav &q = epj[W.jo + e];
                    pp = q.pos;
                    mm = q.mass;
                } else {
                    const sph_spj_monopole &q = spj[W.so + (e - W.nj)];
                    pp = q.pos;
                    mm = q.mass;
                }
                sp[slot(k)] = hi4(pp, o, (float)(G * mm / gscale), &sl[slot(k)], 0.0f);
            }
            __syncthreads();
            const int tc = act ? W.count(tn) : 0;
#pragma unroll 2
            for (int t = 0; t < tc; ++t) {
                const float4 qh = sp[s0 + t], ql = sl[s0 + t];
                const float dx = dfd(ph.x, pl.x, qh.x, ql.x), dy = dfd(ph.y, pl.y, qh.y, ql.y),
                            dz = dfd(ph.z, pl.z, qh.z, ql.z);
                const float ri = rsqrt_a(fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, e2))));
                const float mri = qh.w * ri;
                const float mr3 = mri * ri * ri;
                S.P[0] = fmaf(-mr3, dx, S.P[0]);
                S.P[1] = fmaf(-mr3, dy, S.P[1]);
                S.P[2] = fmaf(-mr3, dz, S.P[2]);
                S.P[3] -= mri;
            }
            if (act) S.add(4 * tile, nl / 32);
            __syncthreads();
        }
        S.store(is[g]);
        __syncthreads();
        if (mine) {
            double D[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) D[k] = total(is[threadIdx.x][k]) * gscale;
            sph_result_grav &out = res[W.io + im];
            out.acc[0] = D[0];
            out.acc[1] = D[1];
            out.acc[2] = D[2];
            out.pot = D[3];
            out.dt = 1.0e30;   // RESULT::Grav::clear(), dt untouched by the functor
        }
        __syncthreads();
    }
}

// blocks of a dispatch: 32 i-particles of a walk each
dim3 walk_grid(int n_walk, int max_i) {
    const int chunks = (max_i + BI - 1) / BI;
    return dim3((unsigned)n_walk, (unsigned)(chunks < 1 ? 1 : (chunks > 4096 ? 4096 : chunks)));
}

}  // namespace

namespace sph {

// launchers for sph_batch.cu, on the tag's stream; max_i: i-particles of the largest walk
void batch32_dens(int n_walk, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_dens *epi,
                  JSrc<sph_epj_dens> epj, sph_result_dens *res) {
    k_walk_dens32<<<walk_grid(n_walk, max_i), BT, 0, st>>>(meta, epi, epj, res);
}
void batch32_drvt(int n_walk, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_drvt *epi,
                  JSrc<sph_epj_drvt> epj, sph_result_drvt *res) {
    k_walk_drvt32<<<walk_grid(n_walk, max_i), BT, 0, st>>>(meta, epi, epj, res);
}
void batch32_hydro(int n_walk, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_hydro *epi,
                   JSrc<sph_epj_hydro> epj, sph_result_hydro *res) {
    k_walk_hydro32<<<walk_grid(n_walk, max_i), BT, 0, st>>>(meta, epi, epj, res);
}
void batch32_grav(int n_walk, int max_i, cudaStream_t st, const int64_t *meta, const sph_epi_grav *epi,
                  JSrc<sph_epj_grav> epj, JSrc<sph_spj_monopole> spj, sph_result_grav *res) {
    k_walk_grav32<<<walk_grid(n_walk, max_i), BT, 0, st>>>(meta, epi, epj, spj, res);
}

}  // namespace sph

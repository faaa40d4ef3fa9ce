// Peel kernels for sm_100a: the drop-in set replacing gpu/peel.cu of
// mwa_hyperdrive (xyzs_to_uvws, rotate, average, iono_loop, subtract_iono,
// add_model).
//
// Differences in shape from the reference (results are the same up to
// rounding): every element-wise kernel runs one thread per (time, channel,
// baseline) so that all SMs are busy and accesses are coalesced (the
// reference runs one thread per baseline with time/channel loops, 32 CTAs at
// 8128 baselines); iono_loop runs all its iterations without host round trips
// -- each iteration is one partial-sum kernel plus one single-CTA update
// kernel that keeps the constants in device memory, and the host reads them
// once at the end (the reference copies them back every iteration,
// peel.cu:709).

#include <vector>

#include "peel.cuh"

namespace hdc {

constexpr int PT = 256;

__global__ void xyzs_to_uvws_kernel(const XYZ* xyzs, const double* lmsts, UVW* uvws, RADec pc, int ntiles, int nbl,
                                    int nt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nbl * nt) return;
    const int t = i / nbl, bl = i % nbl;
    int t1, t2;
    baseline_to_tiles(bl, ntiles, t1, t2);
    const XYZ a = xyzs[(size_t)t * ntiles + t1], b = xyzs[(size_t)t * ntiles + t2];
    const double x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
    double s_ha, c_ha, s_dec, c_dec;
    sincos(pc.dec, &s_dec, &c_dec);
    sincos(lmsts[t] - pc.ra, &s_ha, &c_ha);
    uvws[i] = UVW{s_ha * x + c_ha * y, -s_dec * c_ha * x + s_dec * s_ha * y + c_dec * z,
                  c_dec * c_ha * x - c_dec * s_ha * y + s_dec * z};
}

__device__ __forceinline__ void jf32_mul_f64(JonesF32& j, cplx r) {
    // promote, multiply in f64, demote (peel.cu:78-100)
    const J2 v = load_j32(j) * r;
    j = JonesF32{(float)v.a.re, (float)v.a.im, (float)v.b.re, (float)v.b.im,
                 (float)v.c.re, (float)v.c.im, (float)v.d.re, (float)v.d.im};
}

// JonesF32 * C64 as gpu/common.cuh defines it: the factor is demoted to f32.
__device__ __forceinline__ JonesF32 jf32_mul_c32(const JonesF32& a, cplx r) {
    const float x = (float)r.re, y = (float)r.im;
    return JonesF32{__fsub_rn(__fmul_rn(a.j00_re, x), __fmul_rn(a.j00_im, y)),
                    __fadd_rn(__fmul_rn(a.j00_re, y), __fmul_rn(a.j00_im, x)),
                    __fsub_rn(__fmul_rn(a.j01_re, x), __fmul_rn(a.j01_im, y)),
                    __fadd_rn(__fmul_rn(a.j01_re, y), __fmul_rn(a.j01_im, x)),
                    __fsub_rn(__fmul_rn(a.j10_re, x), __fmul_rn(a.j10_im, y)),
                    __fadd_rn(__fmul_rn(a.j10_re, y), __fmul_rn(a.j10_im, x)),
                    __fsub_rn(__fmul_rn(a.j11_re, x), __fmul_rn(a.j11_im, y)),
                    __fadd_rn(__fmul_rn(a.j11_re, y), __fmul_rn(a.j11_im, x))};
}

// A thread takes ROT_F channels of one (timestep, baseline): its UVWs and
// indices serve them all.  blockIdx.x = baseline block, fastest, then channel
// group, then timestep.
constexpr int ROT_F = 4;
struct VisThread {
    int bl, f0, t;
};
__device__ __forceinline__ VisThread vis_thread(int nbl, int nf) {
    const unsigned nbb = (nbl + PT - 1) / PT, nfg = (nf + ROT_F - 1) / ROT_F;
    return VisThread{(int)(blockIdx.x % nbb) * PT + (int)threadIdx.x, (int)((blockIdx.x / nbb) % nfg) * ROT_F,
                     (int)(blockIdx.x / (nbb * nfg))};
}
static unsigned vis_grid(int nt, int nf, int nbl) {
    return (unsigned)((size_t)((nbl + PT - 1) / PT) * ((nf + ROT_F - 1) / ROT_F) * nt);
}

__global__ void __launch_bounds__(PT) rotate_kernel(JonesF32* vis, int nt, int nbl, int nf, const UVW* from,
                                                    const UVW* to, const double* lambdas) {
    const VisThread x = vis_thread(nbl, nf);
    if (x.bl >= nbl) return;
    const size_t r = (size_t)x.t * nbl + x.bl;
    const double dw = to[r].w - from[r].w;
#pragma unroll
    for (int k = 0; k < ROT_F; k++) {
        const int f = x.f0 + k;
        if (f >= nf) break;
        const size_t i = ((size_t)x.t * nf + f) * nbl + x.bl;
        JonesF32 j = vis[i];
        jf32_mul_f64(j, phasor_turns(-dw / __ldg(lambdas + f)));
        vis[i] = j;
    }
}

__global__ void average_kernel(const JonesF32* hi, const float* w, JonesF32* lo, int nt, int nbl, int nf, int favg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nlo = nf / favg;
    if (i >= nlo * nbl) return;
    const int bl = i % nbl, flo = i / nbl;
    J2 sum = jzero();
    double ws = 0.0;
    for (int t = 0; t < nt; t++)
        for (int fc = flo * favg; fc < flo * favg + favg; fc++) {
            const size_t step = ((size_t)t * nf + fc) * nbl + bl;
            const double wt = w[step];
            sum = sum + load_j32(hi[step]) * wt;
            ws += wt;
        }
    const double d = ws > 0.0 ? ws : 1.0;
    lo[(size_t)flo * nbl + bl] = JonesF32{(float)(sum.a.re / d), (float)(sum.a.im / d), (float)(sum.b.re / d),
                                          (float)(sum.b.im / d),  (float)(sum.c.re / d), (float)(sum.c.im / d),
                                          (float)(sum.d.re / d),  (float)(sum.d.im / d)};
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One iteration's apply + partial sums (peel.cu:437-486 apply_iono and
// iono_loop_kernel, fused with the baseline reduction of reduce_baselines)
// for one (baseline block, channel) of one source; partials [nblk][7] of
// that channel.
__device__ __forceinline__ void iono_partials_body(const JonesF32* resid, const float* weights,
                                                   const JonesF32* model, JonesF32* model_rot, const IonoDev* st,
                                                   const UVW* uvws, const double* lambdas, int nbl, int f,
                                                   int blk, int nblk, double* partials_f) {
    __shared__ double red[PT / 32][7];
    const int bl = blk * PT + threadIdx.x;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    if (bl < nbl) {
        const double u = uvws[bl].u, vv = uvws[bl].v;
        const double arg = -TAU * (u * st->alpha + vv * st->beta);
        double s, c;
        sincos(arg * lambdas[f], &s, &c);
        const size_t step = (size_t)f * nbl + bl;
        const JonesF32 m = jf32_mul_c32(model[step], cplx{c, s} * st->gain);
        model_rot[step] = m;
        const double wt = (double)weights[step];
        const JonesF32 r = resid[step];
        const double ri_re = (double)r.j00_re + (double)r.j11_re;
        const double ri_im = (double)r.j00_im + (double)r.j11_im;
        const double mi_re = (double)m.j00_re + (double)m.j11_re;
        const double mi_im = (double)m.j00_im + (double)m.j11_im;
        const double mr = mi_re * (ri_im - mi_im);
        const double mm = mi_re * mi_re;
        v[0] = wt * mm * u * u;
        v[1] = wt * mm * u * vv;
        v[2] = wt * mm * vv * vv;
        v[3] = wt * mr * u;
        v[4] = wt * mr * vv;
        v[5] = wt * mi_re * ri_re;
        v[6] = wt * mm;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 7; k++) {
        const double s = warp_sum(v[k]);
        if (lane == 0) red[warp][k] = s;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double s = 0.0;
        for (int w = 0; w < PT / 32; w++) s += red[w][threadIdx.x];
        partials_f[(size_t)blk * 7 + threadIdx.x] = s;
    }
}

// grid (ceil(nbl/PT), nf); partials [nf][gridDim.x][7].
__global__ void __launch_bounds__(PT) iono_partials_kernel(const JonesF32* resid, const float* weights,
                                                           const JonesF32* model, JonesF32* model_rot,
                                                           const IonoDev* st, const UVW* uvws, const double* lambdas,
                                                           int nbl, int nf, double* partials) {
    if (st->stop) return;
    iono_partials_body(resid, weights, model, model_rot, st, uvws, lambdas, nbl, blockIdx.y, blockIdx.x, gridDim.x,
                       partials + (size_t)blockIdx.y * gridDim.x * 7);
}

// The constants' update from the seven sums (peel.cu:327-432).
__device__ __forceinline__ void iono_step(const double* t, IonoDev* st, double convergence) {
    const double a_uu = t[0], a_uv = t[1], a_vv = t[2], A_u = t[3], A_v = t[4], s_vm = t[5], s_mm = t[6];
    const double denom = TAU * (a_uu * a_vv - a_uv * a_uv);
    st->alpha += convergence * (A_u * a_vv - A_v * a_uv) / denom;
    st->beta += convergence * (A_v * a_uu - A_u * a_uv) / denom;
    st->gain *= 1. + convergence * (s_vm / s_mm - 1);
    if (st->gain < 0.0) st->stop = 1;  // peel.cu:711
}

// Channel reduction with the lambda scaling and the constants update
// (peel.cu:327-432) for one source; one CTA.
__device__ __forceinline__ void iono_update_body(const double* partials, int nblk, const double* lambdas, int nf,
                                                 IonoDev* st, double convergence) {
    __shared__ double red[PT / 32][7];
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int f = threadIdx.x; f < nf; f += blockDim.x) {
        double s[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int b = 0; b < nblk; b++)
            for (int k = 0; k < 7; k++) s[k] += partials[((size_t)f * nblk + b) * 7 + k];
        const double lam = lambdas[f], lam2 = lam * lam;
        v[0] += s[0] * lam2;
        v[1] += s[1] * lam2;
        v[2] += s[2] * lam2;
        v[3] += s[3] * -lam;
        v[4] += s[4] * -lam;
        v[5] += s[5];
        v[6] += s[6];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < 7; k++) {
        const double s = warp_sum(v[k]);
        if (lane == 0) red[warp][k] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[7];
        for (int k = 0; k < 7; k++) {
            t[k] = 0.0;
            for (int w = 0; w < (int)(blockDim.x / 32); w++) t[k] += red[w][k];
        }
        iono_step(t, st, convergence);
    }
}

__global__ void iono_update_kernel(const double* partials, int nblk, const double* lambdas, int nf, IonoDev* st,
                                   double convergence) {
    if (st->stop) return;
    iono_update_body(partials, nblk, lambdas, nf, st, convergence);
}

__global__ void subtract_iono_kernel(JonesF32* resid, const JonesF32* model, IonoConsts c, IonoConsts old,
                                     const UVW* uvws, const double* lambdas, int nt, int nbl, int nf) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)nt * nf * nbl) return;
    const int bl = (int)(i % nbl);
    const int f = (int)((i / nbl) % nf);
    const int t = (int)(i / ((size_t)nbl * nf));
    const UVW q = uvws[(size_t)t * nbl + bl];
    const double arg = -TAU * (q.u * c.alpha + q.v * c.beta);
    const double old_arg = -TAU * (q.u * old.alpha + q.v * old.beta);
    const double lam = lambdas[f];
    double s, co, so, cold;
    sincos(arg * lam, &s, &co);
    sincos(old_arg * lam, &so, &cold);
    J2 r = load_j32(resid[i]);
    const J2 m = load_j32(model[i]);
    r = r + m * (cplx{cold, so} * old.gain);
    r = r - m * (cplx{co, s} * c.gain);
    resid[i] = JonesF32{(float)r.a.re, (float)r.a.im, (float)r.b.re, (float)r.b.im,
                        (float)r.c.re, (float)r.c.im, (float)r.d.re, (float)r.d.im};
}

__global__ void add_model_kernel(JonesF32* resid, const JonesF32* model, IonoConsts c, const double* lambdas,
                                 const UVW* uvws, int nt, int nf, int nbl) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)nt * nf * nbl) return;
    const int bl = (int)(i % nbl);
    const int f = (int)((i / nbl) % nf);
    const int t = (int)(i / ((size_t)nbl * nf));
    cplx r = {1.0, 0.0};
    if (!(c.alpha == 0.0 && c.beta == 0.0)) {
        const UVW q = uvws[(size_t)t * nbl + bl];
        const double arg = -TAU * (q.u * c.alpha + q.v * c.beta);
        double s, co;
        sincos(arg * lambdas[f], &s, &co);
        r = cplx{co, s};
    }
    const JonesF32 m = jf32_mul_c32(model[i], r * c.gain);
    JonesF32 o = resid[i];
    o.j00_re = __fadd_rn(o.j00_re, m.j00_re);
    o.j00_im = __fadd_rn(o.j00_im, m.j00_im);
    o.j01_re = __fadd_rn(o.j01_re, m.j01_re);
    o.j01_im = __fadd_rn(o.j01_im, m.j01_im);
    o.j10_re = __fadd_rn(o.j10_re, m.j10_re);
    o.j10_im = __fadd_rn(o.j10_im, m.j10_im);
    o.j11_re = __fadd_rn(o.j11_re, m.j11_re);
    o.j11_im = __fadd_rn(o.j11_im, m.j11_im);
    resid[i] = o;
}

static unsigned grid1(size_t n) { return (unsigned)((n + PT - 1) / PT); }

// Host-side body of iono_loop on a stream.
const char* iono_loop_on(const JonesF32* d_resid, const float* d_w, const JonesF32* d_model, JonesF32* d_model_rot,
                         JonesF64* d_fits, IonoConsts* consts, int nbl, int nf, int niter, const UVW* d_uvws,
                         const double* d_lambdas, double convergence, cudaStream_t s) {
    if (nbl <= 0 || nf <= 0) return NULL;
    const int nblk = (nbl + PT - 1) / PT;
    // Layout inside d_fits (nf * nbl JonesF64 = 8 doubles each): partials
    // [nf][nblk][7] first, then the IonoDev block.
    const size_t part_doubles = (size_t)nf * nblk * 7;
    const size_t cap_doubles = (size_t)nf * nbl * 8;
    if (part_doubles + 8 > cap_doubles) return "iono_loop: d_iono_fits too small for this shape";
    double* partials = reinterpret_cast<double*>(d_fits);
    IonoDev* st = reinterpret_cast<IonoDev*>(partials + ((part_doubles + 3) & ~(size_t)3));
    IonoDev h = {consts->alpha, consts->beta, consts->gain, 0, 0};
    HDC_CUDA_RET_STR(cudaMemcpyAsync(st, &h, sizeof(h), cudaMemcpyHostToDevice, s));
    dim3 g(nblk, nf);
    for (int it = 0; it < niter; it++) {
        iono_partials_kernel<<<g, PT, 0, s>>>(d_resid, d_w, d_model, d_model_rot, st, d_uvws, d_lambdas, nbl, nf,
                                              partials);
        count_launches(1);
        iono_update_kernel<<<1, PT, 0, s>>>(partials, nblk, d_lambdas, nf, st, convergence);
        count_launches(1);
    }
    HDC_CUDA_RET_STR(cudaGetLastError());
    HDC_CUDA_RET_STR(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
    HDC_CUDA_RET_STR(cudaStreamSynchronize(s));
    consts->alpha = h.alpha;
    consts->beta = h.beta;
    consts->gain = h.gain;
    return NULL;
}


// One iteration of the fits of a batch of sources from traces (XX + YY; the
// fit reads nothing else): grid (ceil(nbl / IONO_BL), nsrc).  A thread takes one
// baseline and every fourth channel, so u and v leave the channel sums and the
// block reduces 7 numbers once instead of once a channel; the source's last
// block to finish adds the blocks' partials and updates its
// constants.
// Bound: load latency over the short channel loop, then FP64 arithmetic
// (about 36 operations a baseline and channel).  30 sources x 24 channels x
// 8128 baselines: 185 us and a 32 us update kernel an iteration on Jones
// matrices, a reduction per channel; 41 us so.  One source x 12 channels:
// 27 -> 9 us.
constexpr int IONO_BL = 64, IONO_CH = PT / IONO_BL;
__global__ void __launch_bounds__(PT) iono_traces_kernel(const float2* __restrict__ resid, const float* __restrict__ weights,
                                                         const float2* __restrict__ model, IonoDev* states,
                                                         const UVW* __restrict__ uvws, const double* __restrict__ lambdas,
                                                         int nbl, int nf, double* partials, double convergence) {
    const int src = blockIdx.y, nblk = gridDim.x;
    IonoDev* st = states + src;
    if (st->stop) return;
    __shared__ double red[PT / 32][7];
    __shared__ bool last;
    const int bl = blockIdx.x * IONO_BL + threadIdx.x % IONO_BL;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    if (bl < nbl) {
        const UVW q = uvws[(size_t)src * nbl + bl];
        const double turn = -4.0 * (q.u * st->alpha + q.v * st->beta), gain = st->gain;
        double mm2 = 0.0, mr1 = 0.0;  // sums of w mm lambda^2 and w mr lambda
        const float2 *rs = resid + (size_t)src * nf * nbl + bl, *ms = model + (size_t)src * nf * nbl + bl;
        // two channels' loads in flight at a time
        for (int f0 = threadIdx.x / IONO_BL; f0 < nf; f0 += 2 * IONO_CH) {
            float2 r[2], m[2];
            float w[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const size_t i = (size_t)min(f0 + j * IONO_CH, nf - 1) * nbl;
                r[j] = rs[i];
                m[j] = ms[i];
                w[j] = __ldg(weights + i + bl);
            }
#pragma unroll
            for (int j = 0; j < 2; j++) {
                if (f0 + j * IONO_CH >= nf) break;
                const double lam = __ldg(lambdas + f0 + j * IONO_CH);
                const cplx mi = cplx{(double)m[j].x, (double)m[j].y} * (phasor_quarter_f64(turn * lam) * gain);
                const double wm = (double)w[j] * mi.re, mm = wm * mi.re;
                mm2 = fma(mm, lam * lam, mm2);
                mr1 = fma(wm * ((double)r[j].y - mi.im), lam, mr1);
                v[5] = fma(wm, (double)r[j].x, v[5]);
                v[6] += mm;
            }
        }
        v[0] = mm2 * q.u * q.u;
        v[1] = mm2 * q.u * q.v;
        v[2] = mm2 * q.v * q.v;
        v[3] = -mr1 * q.u;
        v[4] = -mr1 * q.v;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 7; k++) {
        const double s = warp_sum(v[k]);
        if (lane == 0) red[warp][k] = s;
    }
    __syncthreads();
    double* part = partials + (size_t)src * nblk * 7;
    if (threadIdx.x < 7) {
        double s = 0.0;
        for (int w = 0; w < PT / 32; w++) s += red[w][threadIdx.x];
        part[(size_t)blockIdx.x * 7 + threadIdx.x] = s;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(&st->pad, 1) == nblk - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    // warp k adds sum k's partials
    if (warp < 7) {
        double s = 0.0;
        for (int b = lane; b < nblk; b += 32) s += __ldcg(part + (size_t)b * 7 + warp);
        s = warp_sum(s);
        if (lane == 0) red[0][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        iono_step(red[0], st, convergence);
        st->pad = 0;
    }
}

size_t iono_partials_bytes(int nsrc, int nbl) {
    return sizeof(double) * (size_t)nsrc * ((nbl + IONO_BL - 1) / IONO_BL) * 7;
}

__global__ void iono_init_kernel(IonoDev* st, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) st[i] = IonoDev{0.0, 0.0, 1.0, 0, 0};
}

cudaError_t iono_states_init(IonoDev* states, int nsrc, cudaStream_t s) {
    iono_init_kernel<<<grid1(nsrc), PT, 0, s>>>(states, nsrc);
    count_launches(1);
    return cudaGetLastError();
}

// The fitted constants, or the old ones where the reference's rule reverts
// them (gpu.rs:541-627); the states are ready for the next fit.
__global__ void iono_result_kernel(IonoDev* st, const IonoConsts* old, IonoConsts* neu, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const IonoConsts o = old[i];
    const IonoConsts c = {o.alpha + st[i].alpha, o.beta + st[i].beta, o.gain * st[i].gain};
    const bool revert = fabs(c.alpha) > 1e-3 || fabs(c.beta) > 1e-3 || c.gain < 0.0 || c.gain > 1.5;
    neu[i] = revert ? o : c;
    st[i] = IonoDev{0.0, 0.0, 1.0, 0, 0};
}

cudaError_t iono_fit(const float2* d_resid, const float* d_w, const float2* d_model, double* d_partials,
                     IonoDev* d_states, const IonoConsts* d_old, IonoConsts* d_neu, int nsrc, int nbl, int nf, int niter,
                     const UVW* d_uvws, const double* d_lambdas, double convergence, cudaStream_t s) {
    if (nbl <= 0 || nf <= 0 || nsrc <= 0) return cudaSuccess;
    const dim3 grid((nbl + IONO_BL - 1) / IONO_BL, nsrc);
    for (int it = 0; it < niter; it++)
        iono_traces_kernel<<<grid, PT, 0, s>>>(d_resid, d_w, d_model, d_states, d_uvws, d_lambdas, nbl, nf, d_partials,
                                               convergence);
    iono_result_kernel<<<grid1(nsrc), PT, 0, s>>>(d_states, d_old, d_neu, nsrc);
    count_launches(niter + 1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The source-by-source loop's two passes over the residual.  They take the
// reference's steps in its order and roundings (rotate to FP32, add_model's
// FP32 product and sum, FP64 averages; rotate, then subtract_iono in FP64)
// without storing what lies between: rotate, two add_models, two averages,
// the copy of the residual and the clears were twelve passes over it.
// ---------------------------------------------------------------------------
// add_model's factor: the ionospheric phasor (exactly 1 when alpha = beta = 0)
// times the gain, as FP32
__device__ __forceinline__ float2 iono_factor(const IonoConsts& c, const UVW& q, double lam) {
    cplx r = {1.0, 0.0};
    if (!(c.alpha == 0.0 && c.beta == 0.0)) r = phasor_turns(-(q.u * c.alpha + q.v * c.beta) * lam);
    return make_float2((float)(r.re * c.gain), (float)(r.im * c.gain));
}
// x y in FP32, each product rounded (JonesF32 * C64 of gpu/common.cuh)
__device__ __forceinline__ float2 mul_rn(float2 x, float2 y) {
    return make_float2(__fsub_rn(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y)),
                       __fadd_rn(__fmul_rn(x.x, y.y), __fmul_rn(x.y, y.x)));
}
__device__ __forceinline__ float2 rotated(float re, float im, cplx r) {
    const cplx v = cplx{(double)re, (double)im} * r;
    return make_float2((float)v.re, (float)v.im);
}

// Weighted means of the traces (XX + YY, which is all that the fit reads) of
// the rotated residual with the source added back and of the source alone:
// 64 bins a CTA, each bin's samples split over 4 threads.
// Bound: the residual's and weights' one pass over memory, then FP64
// arithmetic (two phasors a sample).  4 timesteps x 192 channels x 8128
// baselines: 68 us for what took 680 us in seven launches.
// VEC: the residual is 16-byte aligned (any alignment of float is taken).
template <bool POINT, bool VEC>
__global__ void __launch_bounds__(PT) seq_accumulate_kernel(const SeqArgs A, float2* __restrict__ d_lo,
                                                            float2* __restrict__ m_lo) {
    constexpr int BINS = 64, SPLIT = PT / BINS;
    __shared__ double part[SPLIT - 1][5][BINS];
    const int lane = threadIdx.x % BINS, g = threadIdx.x / BINS;
    const int nlo = A.nf / A.favg;
    const size_t bin = (size_t)blockIdx.x * BINS + lane;
    const bool active = bin < (size_t)nlo * A.nbl;
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // data re, im, model re, im, weight
    if (active) {
        const int bl = (int)(bin % A.nbl), flo = (int)(bin / A.nbl);
        const IonoConsts c = *A.old;
        UVW to;
        double dw = 0.0;
        int tcur = -1;
        for (int k = g; k < A.nt * A.favg; k += SPLIT) {
            const int t = k / A.favg, f = flo * A.favg + k - t * A.favg;
            if (t != tcur) {
                to = A.to[(size_t)t * A.nbl + bl];
                dw = to.w - A.from[(size_t)t * A.nbl + bl].w;
                tcur = t;
            }
            const size_t tf = (size_t)t * A.nf + f, i = tf * A.nbl + bl;
            float2 xx, yy;  // the residual's
            if (VEC) {
                const float4 ra = __ldg(reinterpret_cast<const float4*>(A.resid + i));
                const float4 rb = __ldg(reinterpret_cast<const float4*>(A.resid + i) + 1);
                xx = make_float2(ra.x, ra.y), yy = make_float2(rb.z, rb.w);
            } else {
                const JonesF32* r = A.resid + i;
                xx = make_float2(__ldg(&r->j00_re), __ldg(&r->j00_im));
                yy = make_float2(__ldg(&r->j11_re), __ldg(&r->j11_im));
            }
            const double wt = (double)__ldg(A.w + i), lam = __ldg(A.lam + f);
            float2 mx, my;
            if (POINT) {
                const float4 m = __ldg(A.point + tf);
                mx = make_float2(m.x, 0.f), my = make_float2(m.y, 0.f);
            } else {
                const float4 ma = __ldg(reinterpret_cast<const float4*>(A.model + i));
                const float4 mb = __ldg(reinterpret_cast<const float4*>(A.model + i) + 1);
                mx = make_float2(ma.x, ma.y), my = make_float2(mb.z, mb.w);
            }
            const float2 io = iono_factor(c, to, lam);
            const cplx rot = phasor_turns(-dw / lam);
            mx = mul_rn(mx, io), my = mul_rn(my, io);
            const float2 rx = rotated(xx.x, xx.y, rot), ry = rotated(yy.x, yy.y, rot);
            v[0] = fma(wt, (double)__fadd_rn(rx.x, mx.x) + (double)__fadd_rn(ry.x, my.x), v[0]);
            v[1] = fma(wt, (double)__fadd_rn(rx.y, mx.y) + (double)__fadd_rn(ry.y, my.y), v[1]);
            v[2] = fma(wt, (double)mx.x + (double)my.x, v[2]);
            v[3] = fma(wt, (double)mx.y + (double)my.y, v[3]);
            v[4] += wt;
        }
    }
    if (g > 0)
#pragma unroll
        for (int k = 0; k < 5; k++) part[g - 1][k][lane] = v[k];
    __syncthreads();
    if (g > 0 || !active) return;
#pragma unroll
    for (int q = 0; q < SPLIT - 1; q++)
#pragma unroll
        for (int k = 0; k < 5; k++) v[k] += part[q][k][lane];
    const double d = v[4] > 0.0 ? v[4] : 1.0;
    d_lo[bin] = make_float2((float)(v[0] / d), (float)(v[1] / d));
    m_lo[bin] = make_float2((float)(v[2] / d), (float)(v[3] / d));
}

// The residual into the source's frame with the source re-subtracted:
// rotate, + M iono(old) - M iono(new).
// Bound: FP64 arithmetic (three phasors and three complex products a
// visibility) and, level with it, the residual's two passes over memory (the
// same problem: 127 us; rotate and subtract_iono were 119 + 168 us).
template <bool POINT>
__global__ void __launch_bounds__(PT) seq_update_kernel(const SeqArgs A) {
    const VisThread x = vis_thread(A.nbl, A.nf);
    if (x.bl >= A.nbl) return;
    const UVW q = A.to[(size_t)x.t * A.nbl + x.bl];
    const double dw = q.w - A.from[(size_t)x.t * A.nbl + x.bl].w;
    const IonoConsts old = *A.old, c = *A.neu;
    const double po = -(q.u * old.alpha + q.v * old.beta), pn = -(q.u * c.alpha + q.v * c.beta);
#pragma unroll
    for (int k = 0; k < ROT_F; k++) {
        const int f = x.f0 + k;
        if (f >= A.nf) break;
        const size_t tf = (size_t)x.t * A.nf + f, i = tf * A.nbl + x.bl;
        const double lam = __ldg(A.lam + f);
        JonesF32 j = A.resid[i];
        jf32_mul_f64(j, phasor_turns(-dw / lam));
        J2 m;
        if (POINT) {
            const float4 p = __ldg(A.point + tf);
            m = J2{{(double)p.x, 0.0}, {(double)p.z, (double)p.w}, {(double)p.z, -(double)p.w}, {(double)p.y, 0.0}};
        } else {
            m = load_j32(A.model[i]);
        }
        J2 r = load_j32(j);
        r = r + m * (phasor_turns(po * lam) * old.gain);
        r = r - m * (phasor_turns(pn * lam) * c.gain);
        A.resid[i] = JonesF32{(float)r.a.re, (float)r.a.im, (float)r.b.re, (float)r.b.im,
                              (float)r.c.re, (float)r.c.im, (float)r.d.re, (float)r.d.im};
    }
}

cudaError_t seq_accumulate(const SeqArgs& A, float2* d_lo, float2* m_lo, cudaStream_t s) {
    const unsigned grid = (unsigned)(((size_t)(A.nf / A.favg) * A.nbl + 63) / 64);
    const bool vec = (reinterpret_cast<uintptr_t>(A.resid) & 15) == 0;
    if (A.model)
        vec ? seq_accumulate_kernel<false, true><<<grid, PT, 0, s>>>(A, d_lo, m_lo)
            : seq_accumulate_kernel<false, false><<<grid, PT, 0, s>>>(A, d_lo, m_lo);
    else
        vec ? seq_accumulate_kernel<true, true><<<grid, PT, 0, s>>>(A, d_lo, m_lo)
            : seq_accumulate_kernel<true, false><<<grid, PT, 0, s>>>(A, d_lo, m_lo);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t seq_update(const SeqArgs& A, cudaStream_t s) {
    const unsigned grid = vis_grid(A.nt, A.nf, A.nbl);
    if (A.model)
        seq_update_kernel<false><<<grid, PT, 0, s>>>(A);
    else
        seq_update_kernel<true><<<grid, PT, 0, s>>>(A);
    count_launches(1);
    return cudaGetLastError();
}

// Stream-aware launchers (the drop-in entry points below use stream 0).
cudaError_t k_xyzs_to_uvws(const XYZ* xyzs, const double* lmsts, UVW* uvws, RADec pc, int ntiles, int nbl, int nt,
                           cudaStream_t s) {
    const size_t n = (size_t)nbl * nt;
    if (n == 0) return cudaSuccess;
    xyzs_to_uvws_kernel<<<grid1(n), PT, 0, s>>>(xyzs, lmsts, uvws, pc, ntiles, nbl, nt);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t k_rotate(JonesF32* vis, int nt, int nbl, int nf, const UVW* from, const UVW* to, const double* lambdas,
                     cudaStream_t s) {
    if ((size_t)nt * nf * nbl == 0) return cudaSuccess;
    rotate_kernel<<<vis_grid(nt, nf, nbl), PT, 0, s>>>(vis, nt, nbl, nf, from, to, lambdas);
    count_launches(1);
    return cudaGetLastError();
}

// Low-resolution weights: sum over all timesteps and each channel group,
// clamped at 0 (params/peel/mod.rs:709-755 weights_average).
__global__ void weights_average_kernel(const float* w, float* lo, int nt, int nbl, int nf, int favg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nlo = nf / favg;
    if (i >= nlo * nbl) return;
    const int bl = i % nbl, flo = i / nbl;
    double sum = 0.0;
    for (int t = 0; t < nt; t++)
        for (int fc = flo * favg; fc < flo * favg + favg; fc++) sum += (double)w[((size_t)t * nf + fc) * nbl + bl];
    lo[i] = fmaxf((float)sum, 0.0f);
}

cudaError_t k_weights_average(const float* w, float* lo, int nt, int nbl, int nf, int favg, cudaStream_t s) {
    const size_t n = (size_t)(nf / favg) * nbl;
    if (n == 0) return cudaSuccess;
    weights_average_kernel<<<grid1(n), PT, 0, s>>>(w, lo, nt, nbl, nf, favg);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace hdc

using namespace hdc;

extern "C" const char* xyzs_to_uvws(const XYZ* d_xyzs, const double* d_lmsts, UVW* d_uvws, RADec pointing_centre,
                                    int num_tiles, int num_baselines, int num_timesteps) {
    const size_t n = (size_t)num_baselines * num_timesteps;
    if (n == 0) return NULL;
    xyzs_to_uvws_kernel<<<grid1(n), PT>>>(d_xyzs, d_lmsts, d_uvws, pointing_centre, num_tiles, num_baselines,
                                          num_timesteps);
    count_launches(1);
    HDC_CUDA_RET_STR(cudaGetLastError());
    return NULL;
}

extern "C" const char* rotate(JonesF32* vis_fb, const int num_timesteps, const int num_baselines, const int num_freqs,
                              const UVW* uvws_from, const UVW* uvws_to, const double* lambdas) {
    HDC_CUDA_RET_STR(k_rotate(vis_fb, num_timesteps, num_baselines, num_freqs, uvws_from, uvws_to, lambdas, 0));
    return NULL;
}

extern "C" const char* average(const JonesF32* d_high_res_vis, const float* d_high_res_weights,
                               JonesF32* d_low_res_vis, const int num_timesteps, const int num_baselines,
                               const int num_freqs, const int freq_average_factor) {
    if (freq_average_factor <= 0) return "average: freq_average_factor must be positive";
    const size_t n = (size_t)(num_freqs / freq_average_factor) * num_baselines;
    if (n == 0) return NULL;
    average_kernel<<<grid1(n), PT>>>(d_high_res_vis, d_high_res_weights, d_low_res_vis, num_timesteps, num_baselines,
                                     num_freqs, freq_average_factor);
    count_launches(1);
    HDC_CUDA_RET_STR(cudaGetLastError());
    return NULL;
}

extern "C" const char* iono_loop(const JonesF32* d_vis_residual, const float* d_vis_weights,
                                 const JonesF32* d_vis_model, JonesF32* d_vis_model_rotated, JonesF64* d_iono_fits,
                                 IonoConsts* iono_consts, const int num_baselines, const int num_freqs,
                                 const int num_iterations, const UVW* d_uvws, const double* d_lambdas_m,
                                 const double convergence) {
    return iono_loop_on(d_vis_residual, d_vis_weights, d_vis_model, d_vis_model_rotated, d_iono_fits, iono_consts,
                        num_baselines, num_freqs, num_iterations, d_uvws, d_lambdas_m, convergence, 0);
}

extern "C" const char* subtract_iono(JonesF32* d_vis_residual, const JonesF32* d_vis_model,
                                     const IonoConsts iono_consts, const IonoConsts old_iono_consts, const UVW* d_uvws,
                                     const double* d_lambdas_m, const int num_timesteps, const int num_baselines,
                                     const int num_freqs) {
    const size_t n = (size_t)num_timesteps * num_freqs * num_baselines;
    if (n == 0) return NULL;
    subtract_iono_kernel<<<grid1(n), PT>>>(d_vis_residual, d_vis_model, iono_consts, old_iono_consts, d_uvws,
                                           d_lambdas_m, num_timesteps, num_baselines, num_freqs);
    count_launches(1);
    HDC_CUDA_RET_STR(cudaGetLastError());
    return NULL;
}

extern "C" const char* add_model(JonesF32* d_vis_residual, const JonesF32* d_vis_model, const IonoConsts iono_consts,
                                 const double* d_lambdas_m, const UVW* d_uvws, const int num_timesteps,
                                 const int num_freqs, const int num_baselines) {
    const size_t n = (size_t)num_timesteps * num_freqs * num_baselines;
    if (n == 0) return NULL;
    add_model_kernel<<<grid1(n), PT>>>(d_vis_residual, d_vis_model, iono_consts, d_lambdas_m, d_uvws, num_timesteps,
                                       num_freqs, num_baselines);
    count_launches(1);
    HDC_CUDA_RET_STR(cudaGetLastError());
    return NULL;
}

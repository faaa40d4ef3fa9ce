// Batched peeling: every source's ionospheric fit of a pass from one pass
// over the data (this project's chosen form of peel_gpu,
// params/peel/gpu.rs:25-757).
//
// Source models: a source that is one point component at its own position
// has, in its own frame, the same model on every baseline (phase 1, a beam
// shared by all tiles), so it is kept as one Jones per (timestep, channel);
// any other source's model is materialised at high resolution.
//
// The reference peels sources one after another (Gauss-Seidel): rotate the
// whole high-resolution residual to the source, add the source back, average
// to low resolution, fit (alpha, beta, gain), subtract the re-fitted source,
// move on -- about ten passes over the high-resolution data per source.
// Here a pass fits all sources against the same residual (Jacobi), in the
// phase-centre frame throughout:
//   1. accumulate sweep: for every low-resolution bin and source s,
//        D_s = <w (R rot_s + M_s iono_s(old))>,  Mr_s = <w M_s iono_s(old)>
//      with rot_s = exp(-2 pi i (w_s - w_pc) / lambda) the rotation to the
//      source and <.> the weighted mean over the timeblock and each channel
//      group (the reference's rotate, add_model and vis_average_tfb);
//   2. all sources' iono_loop fits in one launch per iteration
//      (iono_traces_kernel over iono_fit, the reference's arithmetic);
//   3. apply sweep: R += sum_s conj(rot_s) M_s (iono_s(old) - iono_s(new))
//      (the reference's subtract_iono, rotated back).
// Every phase on a baseline is a difference of per-tile phases (uvw_pq =
// uvw_p - uvw_q), so the rotation and ionospheric phasors come from per-tile
// tables [source][timestep][channel][tile] -- 128 phasors where a baseline
// loop would evaluate 8128 -- and a baseline takes tab[p] conj(tab[q]).  Both
// sweeps take 32 x 32 blocks of tile pairs (2 x 2 a thread, on or above the
// diagonal) with the block's 64 rows of the tables in shared memory.
// The fit reads only the traces (XX + YY) of D_s and Mr_s, so the accumulate
// sweep forms only those, from the residual's weighted traces (one complex
// number a sample instead of four), and the fit's low-resolution arrays are
// a quarter as large.
// With one source this is the reference's sequence exactly (up to rounding:
// FP32 products and sums with FP32 phasors after an exact FP64 range
// reduction, as against its f32 intermediates); with several,
// sources
// fitted in the same pass do not see each other's updates until the next
// pass.  The source models M_s (high resolution, source frame) are predicted
// once per timeblock by the modeller and reused by every pass.

#include <algorithm>
#include <cmath>
#include <memory>
#include <mutex>
#include <set>
#include <tuple>
#include <vector>

#include "peel.cuh"

namespace hdc {
namespace pb {

struct SweepArgs {
    JonesF32* resid;        // [nt][nf][nbl], phase-centre frame
    const float* w;         // [nt][nf][nbl]
    float2* wtr;            // [nt][nf][nbl]: w (XX + YY) of the residual
    const JonesF32* models; // [nsrc][nt][nf][nbl], source frames (general sources)
    const float4* ptab;     // [nsrc][nt][nf]: point-at-centre sources' models (xx, yy, Re xy, Im xy; Hermitian), or null
    // per-tile phasors [nsrc][nt][nf][ntiles]; a baseline's factor is
    // tab[p] conj(tab[q]) for its tiles p, q (the phases are differences of
    // per-tile phases, since uvw_pq = uvw_p - uvw_q).  Two phasors a record,
    // (re, re', im, im'), so that both products go through packed arithmetic:
    float4* acc;            // exp(-2 pi i (w_src,p - w_pc,p) / lambda) (rotation to the source frame) and
                            // exp(-2 pi i (alpha u_p + beta v_p) lambda) of the old constants
    float4* app;            // conj(rotation) x the ionospheric phasor of the old and of the new constants
    const IonoConsts* old;  // [nsrc]
    float4* gains;          // [nsrc] (apply sweep): old gain, minus the new one, 1 where no constant changed
    float2* d_lo;           // [nsrc][nlo][nbl] traces of D
    float2* m_lo;           // [nsrc][nlo][nbl] traces of Mr
    int nt, nf, nbl, ntiles, nsrc, favg;
};

// exp(i arg) as (cos, sin): the argument (radians) in FP64, reduced exactly
// in quarter turns, then the FP32 quarter-turn polynomials (< 1 ulp of FP32;
// the residual is stored in FP32, so a per-term phasor error of ~1e-7 is at
// its rounding level)
__device__ __forceinline__ float2 phase_f(double arg) {
    float sn, cs;
    phasor_quarter_f32(arg * 0.63661977236758134308, sn, cs);  // 2 / pi
    return make_float2(cs, sn);
}

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a conj(b)
__device__ __forceinline__ float2 cmulcf(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}

// per-tile UVWs [frame][t][tile] in the frames of the sources (0 .. ns - 1)
// and the phase centre (ns), as xyzs_to_uvws computes them for baselines
__global__ void tile_uvw_kernel(const XYZ* __restrict__ xyz, const double* __restrict__ lmsts,
                                const double2* __restrict__ radec, int nframes, int nt, int ntiles, UVW* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nframes * nt * ntiles) return;
    const int p = i % ntiles, t = (i / ntiles) % nt, fr = i / (ntiles * nt);
    const XYZ a = xyz[(size_t)t * ntiles + p];
    double s_ha, c_ha, s_dec, c_dec;
    sincos(radec[fr].y, &s_dec, &c_dec);
    sincos(lmsts[t] - radec[fr].x, &s_ha, &c_ha);
    out[i] = UVW{s_ha * a.x + c_ha * a.y, -s_dec * c_ha * a.x + s_dec * s_ha * a.y + c_dec * a.z,
                 c_dec * c_ha * a.x - c_dec * s_ha * a.y + s_dec * a.z};
}

// The ionospheric phasor of a tile, exactly 1 when alpha = beta = 0 (as
// add_model skips it).
__device__ __forceinline__ float2 iono_phasor(const IonoConsts& c, const UVW& q, double lam) {
    if (c.alpha == 0.0 && c.beta == 0.0) return make_float2(1.f, 0.f);
    return phase_f(-TAU * (q.u * c.alpha + q.v * c.beta) * lam);
}

// acc[s][t][f][p]: the rotation and the old constants' ionospheric phasor
// (lam: lambda, then 1 / lambda)
__global__ void acc_table_kernel(const UVW* __restrict__ tuvw, const double* __restrict__ lam,
                                 const IonoConsts* __restrict__ k, int ns, int nt, int nf, int ntiles,
                                 float4* __restrict__ acc) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)ns * nt * nf * ntiles) return;
    const int p = (int)(i % ntiles), f = (int)((i / ntiles) % nf), t = (int)((i / ((size_t)ntiles * nf)) % nt);
    const int src = (int)(i / ((size_t)ntiles * nf * nt));
    const UVW q = tuvw[((size_t)src * nt + t) * ntiles + p];
    const double dw = q.w - tuvw[((size_t)ns * nt + t) * ntiles + p].w;
    const float2 r = phase_f(-TAU * dw * lam[nf + f]), io = iono_phasor(k[src], q, lam[f]);
    acc[i] = make_float4(r.x, io.x, r.y, io.y);
}

// app[s][t][f][p] for the fitted constants; acc takes their phasor for the
// next pass.
__global__ void app_table_kernel(const UVW* __restrict__ tuvw, const double* __restrict__ lam,
                                 const IonoConsts* __restrict__ old, const IonoConsts* __restrict__ k, int ns, int nt,
                                 int nf, int ntiles, float4* __restrict__ acc, float4* __restrict__ app,
                                 float4* __restrict__ gains) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (size_t)ns) {
        const IonoConsts a = old[i], b = k[i];
        const bool same = a.alpha == b.alpha && a.beta == b.beta && a.gain == b.gain;
        gains[i] = make_float4((float)a.gain, -(float)b.gain, same ? 1.f : 0.f, 0.f);
    }
    if (i >= (size_t)ns * nt * nf * ntiles) return;
    const int p = (int)(i % ntiles), f = (int)((i / ntiles) % nf), t = (int)((i / ((size_t)ntiles * nf)) % nt);
    const int src = (int)(i / ((size_t)ntiles * nf * nt));
    const float4 a = acc[i];
    const float2 rot = make_float2(a.x, a.z);
    const float2 io = iono_phasor(k[src], tuvw[((size_t)src * nt + t) * ntiles + p], lam[f]);
    const float2 o = cmulcf(make_float2(a.y, a.w), rot), n = cmulcf(io, rot);
    app[i] = make_float4(o.x, n.x, o.y, n.y);
    acc[i] = make_float4(a.x, io.x, a.z, io.y);
}

// w (XX + YY) of every residual sample
__global__ void trace_kernel(const JonesF32* __restrict__ resid, const float* __restrict__ w, size_t n,
                             float2* __restrict__ wtr) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = reinterpret_cast<const float4*>(resid + i)[0], b = reinterpret_cast<const float4*>(resid + i)[1];
    const float wt = w[i];
    wtr[i] = make_float2(wt * (a.x + b.z), wt * (a.y + b.w));
}

// A sweep's block of tile pairs: rows 32 pb .., columns 32 qb .. (blocks on
// or above the diagonal); 256 threads of 2 x 2 pairs, rows and columns 16
// apart.  On the diagonal a thread has two pairs, (row 0, col 0) and (row 1,
// col 1): one of the two half-full diagonal quarters' (below the diagonal of
// the first, the pair (31 - row, 31 - column) of the other) and one of the full
// quarter's.  Four pairs there as well: apply 1.18 ms, two 1.00.
constexpr int TB = 32, NTH = 256;
struct PairBlock {
    int pb, qb;
    int r[2], c[2];  // this thread's row and column slots (columns after the TB rows)
    int bl[4];       // baselines of the pairs (row 0 col 0, row 0 col 1, ..), -1 where none
};
__device__ __forceinline__ PairBlock pair_block(int blk, int ntiles) {
    PairBlock B;
    const int nblk = (ntiles + TB - 1) / TB, noff = nblk * (nblk - 1) / 2;
    if (blk < noff)
        baseline_to_tiles(blk, nblk, B.pb, B.qb);
    else
        B.pb = B.qb = blk - noff;
    const int a = threadIdx.x >> 4, b = threadIdx.x & 15;
    const bool diag = B.pb == B.qb, mirror = diag && a > b;
    B.r[0] = mirror ? 31 - a : a;
    B.c[0] = TB + (mirror ? 31 - b : b);
    B.r[1] = diag ? a : a + 16;
    B.c[1] = TB + b + 16;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int p = B.pb * TB + B.r[i >> 1], q = (B.qb - 1) * TB + B.c[i & 1];
        B.bl[i] = p < q && q < ntiles && !(diag && (i == 1 || i == 2)) ? baseline_index(p, q, ntiles) : -1;
    }
    return B;
}
int pair_blocks(int ntiles) {
    const int nblk = (ntiles + TB - 1) / TB;
    return nblk * (nblk + 1) / 2;
}
// Start copying the record of a block's slot (row tiles, then column tiles)
// from a table row into shared memory; zero past the array.
__device__ __forceinline__ void copy_record(float4* dst, const float4* __restrict__ row, const PairBlock& B, int slot,
                                            int ntiles) {
    const int tile = slot < TB ? B.pb * TB + slot : B.qb * TB + slot - TB;
    const int bytes = tile < ntiles ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(row + (bytes ? tile : 0)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copy_16(float4* dst, const float4* __restrict__ src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest group of this thread's copies have landed
__device__ __forceinline__ void copy_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// Both phasors of a pair from its tiles' records: (re, re') and (im, im') of
// a_p conj(a_q)
__device__ __forceinline__ void pair_phasors(const float4& p, const float4& q, uint64_t& re, uint64_t& im) {
    const uint64_t px = pack2(p.x, p.y), py = pack2(p.z, p.w), nx = pack2(-p.x, -p.y);
    const uint64_t qx = pack2(q.x, q.y), qy = pack2(q.z, q.w);
    re = fma2(py, qy, mul2(px, qx));
    im = fma2(nx, qy, mul2(py, qx));
}

// a Jones matrix as four complex FP32 numbers
struct JF {
    float2 v[4];
};
__device__ __forceinline__ JF load_jf(const JonesF32& j) {
    const float4* p = reinterpret_cast<const float4*>(&j);
    const float4 a = p[0], b = p[1];
    return JF{{make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)}};
}

// The accumulate sweep: traces of D_s and Mr_s of G sources (from blockIdx.x
// G) at the block's pairs and one low-resolution channel.  The tables of
// NSAMP samples are copied while the previous ones are used; a sample and
// source cost a pair two packed products for the two phasors and seven
// multiply-adds.  Products are formed and summed in FP32 (the data are FP32; a
// bin sums nt x favg samples, ~1e-7 relative rounding).
// Bound: issue slots (about 60 % busy at 16 warps an SM, the residual's loads
// read one sample ahead).  30 sources, 8 timesteps x 384 channels x 8128
// baselines: 3.5 ms with all four correlations and a thread per baseline and
// source, 1.16 ms with the groups of sources as the grid's slowest index, 1.13
// as its fastest (a group finds the residual in L2).
constexpr int NSAMP = 4;
template <bool POINTS, int G>
__global__ void __launch_bounds__(NTH, 2) accumulate_kernel(const SweepArgs A) {
    __shared__ alignas(16) float4 s_tab[2][NSAMP][G][2 * TB];
    const PairBlock B = pair_block(blockIdx.y, A.ntiles);
    const int flo = blockIdx.z, nlo = A.nf / A.favg, s0 = blockIdx.x * G;
    const int ng = min(G, A.nsrc - s0), nsamp = A.nt * A.favg;
    const size_t nvis = (size_t)A.nt * A.nf * A.nbl, ntf = (size_t)A.nt * A.nf;
    // samples in order: timestep, then channel of the group; tf = t nf + f
    struct Walk {
        int c, tf;
    };
    auto step = [&](Walk& x) {
        x.tf++;
        if (++x.c == A.favg) x.c = 0, x.tf += A.nf - A.favg;
    };
    const int slot = threadIdx.x & (2 * TB - 1), r0 = threadIdx.x / (2 * TB);
    // this thread's copies: slot's records of the samples (and, G > 1, the
    // source) that its quarter of the CTA takes
    constexpr int NQ = NTH / (2 * TB), KSTEP = G == 1 ? NQ : 1;
    static_assert(G == 1 || G == NQ, "a quarter of the CTA per source, or per sample");
    const int js = G == 1 ? 0 : r0;
    const float4* tab0 = A.acc + (size_t)(s0 + min(js, ng - 1)) * ntf * A.ntiles;
    Walk ws = {0, flo * A.favg};
    if (G == 1)
        for (int e = 0; e < r0; e++) step(ws);
    auto stage = [&](int k0, int buf) {
#pragma unroll
        for (int k = G == 1 ? r0 : 0; k < NSAMP; k += KSTEP) {
            if (js < ng && k0 + k < nsamp) {
                copy_record(&s_tab[buf][k][js][slot], tab0 + (size_t)ws.tf * A.ntiles, B, slot, A.ntiles);
#pragma unroll
                for (int e = 0; e < KSTEP; e++) step(ws);
            }
        }
        copy_commit();
    };
    float2 nr[4];
    float nw[4];
    Walk wf = {0, flo * A.favg};
    auto fetch = [&](int k) {
        const size_t row = (size_t)wf.tf * A.nbl;
        const float2* pr = A.wtr + row;
        const float* pw = A.w + row;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool has = k < nsamp && B.bl[i] >= 0;
            nr[i] = has ? __ldg(pr + B.bl[i]) : make_float2(0.f, 0.f);
            nw[i] = has ? __ldg(pw + B.bl[i]) : 0.f;
        }
        step(wf);
    };
    stage(0, 0);
    fetch(0);
    float g[G];
#pragma unroll
    for (int j = 0; j < G; j++) g[j] = j < ng ? (float)A.old[s0 + j].gain : 0.f;
    float2 sd[4][G], sm[4][G];
    float sw[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < G; j++) sd[i][j] = sm[i][j] = make_float2(0.f, 0.f);
    Walk wk = {0, flo * A.favg};
    for (int k0 = 0; k0 < nsamp; k0 += NSAMP) {
        const int n = min(NSAMP, nsamp - k0), buf = (k0 / NSAMP) & 1;
        stage(k0 + NSAMP, buf ^ 1);
        copy_wait_one();
        __syncthreads();
        for (int k = 0; k < n; k++) {
            const size_t tf = wk.tf, row = tf * A.nbl;
            step(wk);
            float2 r[4];
            float w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) r[i] = nr[i], w[i] = nw[i], sw[i] += w[i];
            fetch(k0 + k + 1);  // the next sample's, in flight during this one
#pragma unroll
            for (int j = 0; j < G; j++) {
                if (j >= ng) break;
                float gm = g[j];
                if (POINTS) {
                    const float2 m = __ldg(reinterpret_cast<const float2*>(A.ptab + (size_t)(s0 + j) * ntf + tf));
                    gm *= m.x + m.y;
                }
                const float4(&tab)[2 * TB] = s_tab[buf][k][j];
                const float4 p[2] = {tab[B.r[0]], tab[B.r[1]]}, q[2] = {tab[B.c[0]], tab[B.c[1]]};
                auto pair = [&](int i) {
                    uint64_t re2, im2;
                    pair_phasors(p[i >> 1], q[i & 1], re2, im2);
                    const float2 re = unpack2(re2), im = unpack2(im2);  // rotation, ionosphere
                    sd[i][j].x = fmaf(r[i].x, re.x, fmaf(-r[i].y, im.x, sd[i][j].x));
                    sd[i][j].y = fmaf(r[i].x, im.x, fmaf(r[i].y, re.x, sd[i][j].y));
                    const float c = w[i] * gm;
                    if (POINTS) {
                        sm[i][j].x = fmaf(c, re.y, sm[i][j].x);
                        sm[i][j].y = fmaf(c, im.y, sm[i][j].y);
                    } else if (B.bl[i] >= 0) {
                        const float4* mp = reinterpret_cast<const float4*>(A.models + (size_t)(s0 + j) * nvis + row + B.bl[i]);
                        const float4 m0 = __ldg(mp), m1 = __ldg(mp + 1);
                        const float2 cm = make_float2(c * (m0.x + m1.z), c * (m0.y + m1.w));
                        sm[i][j].x = fmaf(cm.x, re.y, fmaf(-cm.y, im.y, sm[i][j].x));
                        sm[i][j].y = fmaf(cm.x, im.y, fmaf(cm.y, re.y, sm[i][j].y));
                    }
                };
                pair(0);
                pair(3);
                if (B.pb != B.qb) pair(1), pair(2);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (B.bl[i] < 0) continue;
        const double inv = 1.0 / (sw[i] > 0.f ? (double)sw[i] : 1.0);
#pragma unroll
        for (int j = 0; j < G; j++) {
            if (j >= ng) break;
            const size_t o = ((size_t)(s0 + j) * nlo + flo) * A.nbl + B.bl[i];
            A.d_lo[o] = make_float2((float)((sd[i][j].x + sm[i][j].x) * inv), (float)((sd[i][j].y + sm[i][j].y) * inv));
            A.m_lo[o] = make_float2((float)(sm[i][j].x * inv), (float)(sm[i][j].y * inv));
        }
    }
}

// The apply sweep: all sources' updates at the block's pairs of TFS
// consecutive (timestep, channel) rows, summed in FP32 and added to the
// residual once:
//   R += sum_s M_s conj(rot_s) (g_old io_old - g_new io_new)
// and, where a further sub-batch follows (next), its weighted trace.  A point
// source's M is Hermitian: with M_xy = a + i b the sums of m_xx z, m_yy z, a z
// and b z give XY = P + i Q, YX = P - i Q.  The tables of SCHUNK sources are
// copied while the previous ones are used, across rows.
// Bound: issue slots and, below them, the residual's two passes over memory
// (0.3 ms).  The same problem: 2.97 ms with a thread per baseline, 1.00 ms so.
constexpr int SCHUNK = 16, TFS = 8;
template <bool POINTS>
__global__ void __launch_bounds__(NTH, 2) apply_kernel(const SweepArgs A, bool next) {
    __shared__ alignas(16) float4 s_tab[2][SCHUNK][2 * TB];
    __shared__ alignas(16) float4 s_m[2][SCHUNK], s_g[2][SCHUNK];
    const int nblk = (A.ntiles + TB - 1) / TB, nblocks = nblk * (nblk + 1) / 2;
    const PairBlock B = pair_block(blockIdx.x % nblocks, A.ntiles);
    const size_t ntf = (size_t)A.nt * A.nf, tf0 = (size_t)(blockIdx.x / nblocks) * TFS;
    const int rows = (int)min((size_t)TFS, ntf - tf0), nch = (A.nsrc + SCHUNK - 1) / SCHUNK, steps = rows * nch;
    const int slot = threadIdx.x & (2 * TB - 1), r0 = threadIdx.x / (2 * TB);
    auto stage = [&](int st, int buf) {
        if (st < steps) {
            const int s0 = (st % nch) * SCHUNK;
            const float4* row = A.app + ((size_t)s0 * ntf + tf0 + st / nch) * A.ntiles;
            const int n = min(SCHUNK, A.nsrc - s0);
            for (int j = r0; j < n; j += NTH / (2 * TB))
                copy_record(&s_tab[buf][j][slot], row + (size_t)j * ntf * A.ntiles, B, slot, A.ntiles);
            const int j = threadIdx.x % SCHUNK;
            if (threadIdx.x < SCHUNK && j < n)
                copy_16(&s_g[buf][j], A.gains + s0 + j);
            else if (POINTS && threadIdx.x < 2 * SCHUNK && j < n)
                copy_16(&s_m[buf][j], A.ptab + (size_t)(s0 + j) * ntf + tf0 + st / nch);
        }
        copy_commit();
    };
    stage(0, 0);
    uint64_t acc[4][4];
    float4 ra[4], rb[4];
    for (int st = 0; st < steps; st++) {
        const int chunk = st % nch, s0 = chunk * SCHUNK, n = min(SCHUNK, A.nsrc - s0);
        const size_t tf = tf0 + st / nch, row = tf * A.nbl;
        if (chunk == 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
#pragma unroll
                for (int e = 0; e < 4; e++) acc[i][e] = 0;
                // the row's residual, in flight while its sources are summed
                const float4* r = reinterpret_cast<const float4*>(A.resid + row + max(B.bl[i], 0));
                ra[i] = r[0];
                rb[i] = r[1];
            }
        }
        stage(st + 1, (st + 1) & 1);
        copy_wait_one();
        __syncthreads();
        for (int j = 0; j < n; j++) {
            const float4 gn = s_g[st & 1][j];
            if (gn.z != 0.f) continue;  // its constants did not change
            const float4(&tab)[2 * TB] = s_tab[st & 1][j];
            const float4 p[2] = {tab[B.r[0]], tab[B.r[1]]}, q[2] = {tab[B.c[0]], tab[B.c[1]]};
            const uint64_t gg = pack2(gn.x, gn.y);
            uint64_t wm[4];
            if (POINTS) {
                const float4 m = s_m[st & 1][j];
                wm[0] = dup2(m.x), wm[1] = dup2(m.y), wm[2] = dup2(m.z), wm[3] = dup2(m.w);
            }
            auto pair = [&](int i) {
                uint64_t re2, im2;
                pair_phasors(p[i >> 1], q[i & 1], re2, im2);
                const float2 re = unpack2(mul2(re2, gg)), im = unpack2(mul2(im2, gg));
                const float2 z = make_float2(re.x + re.y, im.x + im.y);
                if (POINTS) {
                    const uint64_t z2 = pack2(z.x, z.y);
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[i][e] = fma2(wm[e], z2, acc[i][e]);
                } else if (B.bl[i] >= 0) {
                    const JF m = load_jf(A.models[(size_t)(s0 + j) * ntf * A.nbl + row + B.bl[i]]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float2 c = cmulf(m.v[e], z), o = unpack2(acc[i][e]);
                        acc[i][e] = pack2(o.x + c.x, o.y + c.y);
                    }
                }
            };
            pair(0);
            pair(3);
            if (B.pb != B.qb) pair(1), pair(2);
        }
        __syncthreads();
        if (chunk != nch - 1) continue;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (B.bl[i] < 0) continue;
            const float2 c0 = unpack2(acc[i][0]), c1 = unpack2(acc[i][1]), c2 = unpack2(acc[i][2]), c3 = unpack2(acc[i][3]);
            // general sources keep the four correlations in their order
            const float2 xx = c0, yy = POINTS ? c1 : c3;
            const float2 xy = POINTS ? make_float2(c2.x - c3.y, c2.y + c3.x) : c1;
            const float2 yx = POINTS ? make_float2(c2.x + c3.y, c2.y - c3.x) : c2;
            const float4 a = ra[i], b = rb[i];
            const float4 na = make_float4(a.x + xx.x, a.y + xx.y, a.z + xy.x, a.w + xy.y);
            const float4 nb = make_float4(b.x + yx.x, b.y + yx.y, b.z + yy.x, b.w + yy.y);
            float4* r = reinterpret_cast<float4*>(A.resid + row + B.bl[i]);
            r[0] = na;
            r[1] = nb;
            if (next) {
                const float wt = __ldg(A.w + row + B.bl[i]);
                A.wtr[row + B.bl[i]] = make_float2(wt * (na.x + nb.z), wt * (na.y + nb.w));
            }
        }
    }
}

std::mutex g_tune_mu;
std::set<std::tuple<int, int, int, int, int>> g_seen;  // shapes (nt, nf, nbl, nsrc, favg) timed
struct Tuning {
    int bx = 0, sy = 0;
    float ms = 0.f;
} g_last;

template <bool POINTS, int G>
void launch_acc(const SweepArgs& A, cudaStream_t s) {
    const dim3 grid((A.nsrc + G - 1) / G, pair_blocks(A.ntiles), A.nf / A.favg);
    accumulate_kernel<POINTS, G><<<grid, NTH, 0, s>>>(A);
    count_launches(1);
}

// The accumulate sweep: GRP sources a thread share its residual loads where
// that leaves two CTAs for every SM, else one.  The first sweep of a problem
// shape is timed (hdc_peel_batched_tuning reports it).
constexpr int GRP = 4;
cudaError_t accumulate(const SweepArgs& A, cudaStream_t s) {
    const long long ctas = (long long)pair_blocks(A.ntiles) * (A.nf / A.favg) * ((A.nsrc + GRP - 1) / GRP);
    int dev = 0, nsm = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const bool group = ctas >= 2 * nsm;
    bool timed;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        timed = g_seen.insert(std::make_tuple(A.nt, A.nf, A.nbl, A.nsrc, A.favg)).second;
    }
    cudaEvent_t a = nullptr, b = nullptr;
    if (timed) {
        cudaEventCreate(&a);
        cudaEventCreate(&b);
        cudaEventRecord(a, s);
    }
    if (A.ptab)
        group ? launch_acc<true, GRP>(A, s) : launch_acc<true, 1>(A, s);
    else
        group ? launch_acc<false, GRP>(A, s) : launch_acc<false, 1>(A, s);
    cudaError_t e = cudaGetLastError();
    if (timed) {
        float ms = 0.f;
        cudaEventRecord(b, s);
        if (e == cudaSuccess) e = cudaEventSynchronize(b);
        if (e == cudaSuccess) cudaEventElapsedTime(&ms, a, b);
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_last = Tuning{NTH, 1, ms};
    }
    return e;
}

void apply(const SweepArgs& A, bool next, cudaStream_t s) {
    const unsigned grid = (unsigned)((size_t)pair_blocks(A.ntiles) * (((size_t)A.nt * A.nf + TFS - 1) / TFS));
    if (A.ptab)
        apply_kernel<true><<<grid, NTH, 0, s>>>(A, next);
    else
        apply_kernel<false><<<grid, NTH, 0, s>>>(A, next);
    count_launches(1);
}

}  // namespace pb
}  // namespace hdc

using namespace hdc;

#define PB_CK(call)                                                                    \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess) {                                                       \
            cudaGetLastError();                                                        \
            set_error("hdc_peel_timeblock_batched: %s: %s", #call, cudaGetErrorString(e_)); \
            return e_ == cudaErrorMemoryAllocation ? HDC_ERR_ALLOC : HDC_ERR_CUDA;     \
        }                                                                              \
    } while (0)

extern "C" int hdc_peel_timeblock_batched(JonesF32* d_resid_tfb, const float* d_weights_tfb, int num_timesteps,
                                          int num_freqs, const double* h_freqs, const XYZ* h_tile_xyzs, int num_tiles,
                                          const double* h_lmsts, double average_lmst, RADec phase_centre,
                                          int num_sources, const HdcSkyModel* h_sources,
                                          const RADec* h_source_positions, IonoConsts* h_iono_consts,
                                          const HdcPeelParams* params, hdcStream_t stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (!d_resid_tfb || !d_weights_tfb || !h_freqs || !h_tile_xyzs || !h_lmsts || !params || num_tiles < 2 ||
        num_timesteps < 1 || num_freqs < 1 || num_sources < 0 ||
        (num_sources > 0 && (!h_sources || !h_iono_consts || !h_source_positions))) {
        set_error("hdc_peel_timeblock_batched: invalid arguments");
        return HDC_ERR_ARG;
    }
    const int favg = params->freq_average_factor;
    if (favg < 1 || num_freqs % favg != 0) {
        set_error("hdc_peel_timeblock_batched: %d channels are not a multiple of the averaging factor %d", num_freqs,
                  favg);
        return HDC_ERR_ARG;
    }
    if (reinterpret_cast<uintptr_t>(d_resid_tfb) & 15) {
        set_error("hdc_peel_timeblock_batched: the residual's address is not a multiple of 16 bytes");
        return HDC_ERR_ARG;
    }
    if (num_sources == 0) return HDC_OK;
    const int nt = num_timesteps, nf = num_freqs, nbl = num_tiles * (num_tiles - 1) / 2, nlo = nf / favg;
    const int ns = num_sources;
    const size_t nvis = (size_t)nt * nf * nbl;

    std::vector<double> lam(2 * (size_t)nf), lam_lo(nlo);
    for (int f = 0; f < nf; f++) lam[f] = VEL_C / h_freqs[f];
    for (int f = 0; f < nf; f++) lam[nf + f] = 1.0 / lam[f];
    for (int k = 0; k < nlo; k++) {
        double sum = 0.0;
        for (int f = k * favg; f < (k + 1) * favg; f++) sum += h_freqs[f];
        lam_lo[k] = VEL_C / (sum / favg);
    }
    std::vector<XYZ> xyz_t((size_t)nt * num_tiles);
    for (int t = 0; t < nt; t++)
        for (int i = 0; i < num_tiles; i++) xyz_t[(size_t)t * num_tiles + i] = h_tile_xyzs[i];

    // point-at-centre sources keep a (timestep, channel) table; otherwise
    // the models need ns x nvis JonesF32 of device memory
    // (with a beam shared by all tiles, or none: per-tile beams make a
    // point's model depend on the baseline)
    const bool points = peel_point_sources(h_sources, h_source_positions, ns, params->beam_kind);
    const size_t need = points ? sizeof(float4) * (size_t)ns * nt * nf : sizeof(JonesF32) * nvis * (size_t)ns;
    const size_t ntab = (size_t)ns * nt * nf * num_tiles;  // per-tile phasor tables
    // one sub-batch's apply table at a time
    const int batch = params->batch_size > 0 ? std::min(params->batch_size, ns) : ns;
    // the call's larger buffers: models, phasor tables, traces and
    // low-resolution sums, UVWs (what the pool holds idle serves them too)
    const size_t buffers = need + sizeof(float4) * (ntab + (size_t)batch * nt * nf * num_tiles) + sizeof(float2) * nvis +
                           sizeof(float2) * 2 * (size_t)batch * nlo * nbl + iono_partials_bytes(batch, nbl) +
                           sizeof(UVW) * ((size_t)ns * nbl + (points ? 0 : (size_t)ns * nt * nbl));
    size_t free_b = 0, total_b = 0;
    PB_CK(cudaMemGetInfo(&free_b, &total_b));
    free_b += pool_idle_bytes();
    if (std::max(buffers, need + (size_t)(1u << 30)) > free_b) {
        set_error("hdc_peel_timeblock_batched: %d sources need %zu MB of device memory (models %zu MB), %zu MB free", ns,
                  buffers >> 20, need >> 20, free_b >> 20);
        return HDC_ERR_ALLOC;
    }
    DevBuf b_tuvw, b_radec, b_acc, b_app, b_wtr;
    DevBuf b_lam, b_lam_lo, b_lmst, b_avg_lmst, b_xyz, b_uv_src, b_uv_lo, b_models, b_dlo, b_mlo, b_wlo, b_part,
        b_st, b_consts, b_gains;
    PB_CK(b_lam.alloc(sizeof(double) * 2 * nf, s));  // lambda, then 1 / lambda
    PB_CK(b_lam_lo.alloc(sizeof(double) * nlo, s));
    PB_CK(b_lmst.alloc(sizeof(double) * nt, s));
    PB_CK(b_avg_lmst.alloc(sizeof(double), s));
    PB_CK(b_xyz.alloc(sizeof(XYZ) * xyz_t.size(), s));
    if (!points) PB_CK(b_uv_src.alloc(sizeof(UVW) * (size_t)ns * nt * nbl, s));
    PB_CK(b_tuvw.alloc(sizeof(UVW) * (size_t)(ns + 1) * nt * num_tiles, s));
    PB_CK(b_radec.alloc(sizeof(double2) * (ns + 1), s));
    PB_CK(b_acc.alloc(sizeof(float4) * ntab, s));
    PB_CK(b_app.alloc(sizeof(float4) * (size_t)batch * nt * nf * num_tiles, s));
    PB_CK(b_wtr.alloc(sizeof(float2) * nvis, s));
    PB_CK(b_uv_lo.alloc(sizeof(UVW) * (size_t)ns * nbl, s));
    PB_CK(points ? b_models.alloc(need, s) : b_models.alloc_plain(need));
    PB_CK(b_dlo.alloc(sizeof(float2) * (size_t)batch * nlo * nbl, s));
    PB_CK(b_mlo.alloc(sizeof(float2) * (size_t)batch * nlo * nbl, s));
    PB_CK(b_wlo.alloc(sizeof(float) * (size_t)nlo * nbl, s));
    PB_CK(b_part.alloc(iono_partials_bytes(batch, nbl), s));
    PB_CK(b_st.alloc(sizeof(IonoDev) * batch, s));
    PB_CK(b_consts.alloc(sizeof(IonoConsts) * 2 * ns, s));  // a pass's old and new constants, then the other way round
    PB_CK(b_gains.alloc(sizeof(float4) * batch, s));
    PB_CK(cudaMemcpyAsync(b_lam.p, lam.data(), sizeof(double) * 2 * nf, cudaMemcpyHostToDevice, s));
    PB_CK(cudaMemcpyAsync(b_lam_lo.p, lam_lo.data(), sizeof(double) * nlo, cudaMemcpyHostToDevice, s));
    PB_CK(cudaMemcpyAsync(b_lmst.p, h_lmsts, sizeof(double) * nt, cudaMemcpyHostToDevice, s));
    PB_CK(cudaMemcpyAsync(b_avg_lmst.p, &average_lmst, sizeof(double), cudaMemcpyHostToDevice, s));
    PB_CK(cudaMemcpyAsync(b_xyz.p, xyz_t.data(), sizeof(XYZ) * xyz_t.size(), cudaMemcpyHostToDevice, s));
    PB_CK(k_weights_average(d_weights_tfb, b_wlo.as<float>(), nt, nbl, nf, favg, s));
    // per-tile UVWs in every source's frame and the phase centre's, the
    // rotation phasors to each source (fixed for the timeblock) with the given
    // constants' ionospheric ones, and the residual's weighted traces
    std::vector<double2> radec(ns + 1);
    for (int i = 0; i < ns; i++) radec[i] = make_double2(h_source_positions[i].ra, h_source_positions[i].dec);
    radec[ns] = make_double2(phase_centre.ra, phase_centre.dec);
    PB_CK(cudaMemcpyAsync(b_radec.p, radec.data(), sizeof(double2) * (ns + 1), cudaMemcpyHostToDevice, s));
    PB_CK(cudaMemcpyAsync(b_consts.p, h_iono_consts, sizeof(IonoConsts) * ns, cudaMemcpyHostToDevice, s));
    PB_CK(iono_states_init(b_st.as<IonoDev>(), batch, s));
    {
        const int n = (ns + 1) * nt * num_tiles;
        pb::tile_uvw_kernel<<<(n + 255) / 256, 256, 0, s>>>(b_xyz.as<XYZ>(), b_lmst.as<double>(),
                                                            b_radec.as<double2>(), ns + 1, nt, num_tiles,
                                                            b_tuvw.as<UVW>());
        pb::acc_table_kernel<<<(unsigned)((ntab + 255) / 256), 256, 0, s>>>(
            b_tuvw.as<UVW>(), b_lam.as<double>(), b_consts.as<IonoConsts>(), ns, nt, nf, num_tiles, b_acc.as<float4>());
        pb::trace_kernel<<<(unsigned)((nvis + 255) / 256), 256, 0, s>>>(d_resid_tfb, d_weights_tfb, nvis,
                                                                       b_wtr.as<float2>());
        count_launches(3);
        PB_CK(cudaGetLastError());
    }
    // per source: UVWs in its frame and its high-resolution model (once per
    // timeblock)
    for (int i = 0; i < ns; i++) {
        if (!points)
            PB_CK(k_xyzs_to_uvws(b_xyz.as<XYZ>(), b_lmst.as<double>(), b_uv_src.as<UVW>() + (size_t)i * nt * nbl,
                                 h_source_positions[i], num_tiles, nbl, nt, s));
        PB_CK(k_xyzs_to_uvws(b_xyz.as<XYZ>(), b_avg_lmst.as<double>(), b_uv_lo.as<UVW>() + (size_t)i * nbl,
                             h_source_positions[i], num_tiles, nbl, 1, s));
    }
    if (points) {
        const int rc = peel_point_table(h_sources, ns, h_freqs, nf, h_lmsts, nt, params->array_latitude_rad,
                                        params->beam_kind, b_models.as<float4>(), s);
        if (rc) return rc;
    } else {
        PB_CK(cudaMemsetAsync(b_models.p, 0, need, s));
        for (int i = 0; i < ns; i++) {
            HdcModeller* hm = nullptr;
            int rc = peel_modeller_new(&h_sources[i], h_tile_xyzs, num_tiles, h_freqs, num_freqs,
                                       h_source_positions[i], params, &hm);
            if (rc) return rc;
            std::unique_ptr<Modeller> m(reinterpret_cast<Modeller*>(hm));
            const UVW* uv = b_uv_src.as<UVW>() + (size_t)i * nt * nbl;
            for (int t = 0; t < nt; t++) {
                rc = m->model_uvws(h_lmsts[t], uv + (size_t)t * nbl,
                                   b_models.as<JonesF32>() + (size_t)i * nvis + (size_t)t * nf * nbl, s);
                if (rc) return rc;
            }
        }
    }

    pb::SweepArgs A;
    A.resid = d_resid_tfb;
    A.w = d_weights_tfb;
    A.wtr = b_wtr.as<float2>();
    A.models = points ? nullptr : b_models.as<JonesF32>();
    A.ptab = points ? b_models.as<float4>() : nullptr;
    A.acc = b_acc.as<float4>();
    A.app = b_app.as<float4>();
    A.gains = b_gains.as<float4>();
    A.d_lo = b_dlo.as<float2>();
    A.m_lo = b_mlo.as<float2>();
    A.nt = nt;
    A.nf = nf;
    A.nbl = nbl;
    A.ntiles = num_tiles;
    A.nsrc = ns;
    A.favg = favg;
    // sources in sub-batches of `batch` in list order: within a sub-batch the
    // fits share the residual (Jacobi); each sub-batch sees the residual the
    // earlier ones left (the reference's Gauss-Seidel order between them)
    const IonoConsts* result = b_consts.as<IonoConsts>();
    for (int pass = 0; pass < params->num_passes; pass++) {
        const IonoConsts* old = b_consts.as<IonoConsts>() + (pass & 1) * ns;
        IonoConsts* neu = b_consts.as<IonoConsts>() + ((pass + 1) & 1) * ns;
        for (int b0 = 0; b0 < ns; b0 += batch) {
            const int nb = std::min(batch, ns - b0);
            const size_t ntab_b = (size_t)nb * nt * nf * num_tiles;
            pb::SweepArgs B = A;
            B.nsrc = nb;
            B.models = A.models ? A.models + (size_t)b0 * nvis : nullptr;
            B.ptab = A.ptab ? A.ptab + (size_t)b0 * nt * nf : nullptr;
            B.acc = A.acc + (size_t)b0 * nt * nf * num_tiles;
            B.old = old + b0;
            PB_CK(pb::accumulate(B, s));
            PB_CK(iono_fit(B.d_lo, b_wlo.as<float>(), B.m_lo, b_part.as<double>(), b_st.as<IonoDev>(), old + b0,
                           neu + b0, nb, nbl, nlo, params->num_loops, b_uv_lo.as<UVW>() + (size_t)b0 * nbl,
                           b_lam_lo.as<double>(), params->convergence, s));
            // app from tuvw rows of this sub-batch's sources
            pb::app_table_kernel<<<(unsigned)((ntab_b + 255) / 256), 256, 0, s>>>(
                b_tuvw.as<UVW>() + (size_t)b0 * nt * num_tiles, b_lam.as<double>(), old + b0, neu + b0, nb, nt, nf,
                num_tiles, B.acc, B.app, B.gains);
            count_launches(1);
            PB_CK(cudaGetLastError());
            pb::apply(B, pass + 1 < params->num_passes || b0 + batch < ns, s);
            PB_CK(cudaGetLastError());
        }
        result = neu;
    }
    PB_CK(cudaMemcpyAsync(h_iono_consts, result, sizeof(IonoConsts) * ns, cudaMemcpyDeviceToHost, s));
    PB_CK(cudaStreamSynchronize(s));
    return HDC_OK;
}

extern "C" int hdc_peel_batched_tuning(int* block_bins, int* block_sources, float* ms) {
    std::lock_guard<std::mutex> lk(pb::g_tune_mu);
    if (block_bins) *block_bins = pb::g_last.bx;
    if (block_sources) *block_sources = pb::g_last.sy;
    if (ms) *ms = pb::g_last.ms;
    return HDC_OK;
}

// The native modeller's FP64 predict (HDC_PREDICT_DIRECT), factored by tile.
//
// A native modeller's baseline UVW is a tile difference (uvw_pq = uvw_p -
// uvw_q), so the phasor of a term factors: exp(2 pi i t_pq) = A_p conj(A_q)
// with A_p = exp(2 pi i (u_p l + v_p m + w_p (n - 1))), and an envelope's
// coordinates are differences of per-tile ones.  A CTA takes a block of tile
// pairs of one channel (on or above the diagonal) and, per staged chunk of
// components, forms in shared memory its tiles' phasors (and Gaussian or
// shapelet coordinates); its 256 threads then take the pairs, so one FP64
// sincos serves 16 baselines (32 x 32 pairs, 2 x 2 a thread) or 8 (16 x 16, one
// a thread) and a pair costs a complex product (4 operations) instead of a
// sincos.  whole_tiles says which blocks.
//
// Shared beam (or none): W = B S B^H is Hermitian, so with W_xy = a + i b the
// four correlations come from the sums of w_xx z, w_yy z, a z and b z (8
// fused multiply-adds a term; XY = P + i Q and YX = P - i Q at the end).
// Per-tile beams: M_p = A_p B_p S and N_q = A_q B_q are formed per tile, and
// a term is M_p N_q^H (32 fused multiply-adds).
//
// Bound: the FP64 pipe (64 lanes per clock and SM; 0.64 busy over the points'
// sweep and tables) and, level with it, shared-memory reads (96 bytes a lane
// and component of the four pairs, 128 bytes a clock).  128 tiles x 384
// channels x 1000 points: 13.2 ms with a thread per baseline, 4.3 with the
// library's sincospi, 4.0 with this kernel's polynomials (1 x 2 pairs a thread
// 4.3, 4 x 2 at half the warps 4.8), 3.7 with a diagonal block's two half-full
// quarters summed as one, 3.5 with those blocks last.  Every value is FP64,
// tile positions are taken from the array's centroid (so a tile's phase is no
// larger than its baselines'), and sums run over the components in order.
// The drop-in calls keep the per-baseline kernel (predict.cu): their UVWs
// are the caller's and need not be tile differences.  So do one or two
// components, which do not pay for the tables (launch_direct).

#include <atomic>
#include <type_traits>

#include "predict.cuh"

namespace hdc {
namespace pairs {

constexpr int NTH = 256;  // threads of a CTA, 16 x 16
constexpr int GRP = 32;   // table slots a CTA of single pairs has (rows, then columns)

// The tile pairs of a CTA (us per call, 65 tiles x 128 channels x 200, with a
// thread per baseline and its own phasors / in 32 x 32 blocks only / so: FP64
// Gaussians 389 / 404 / 268, the chosen form's 127 / 197 / 139, with per-tile
// beams 379 / 587 / 400).  H 2: a block of 32 x 32 pairs of groups of 32 tiles,
// on or above the diagonal; a thread takes 2 x 2 of them, 16 apart.  (The last
// group may reach past the array: its places there repeat the last tile.)  H 1: at
// most 256 pairs, one a thread: blocks of 16 x 16 of whole groups of 16 (a
// diagonal block's 120 pairs counted), and strips of the last tiles, fewer than
// 16, with as many others as fit the table slots (their pairs counted too).  Pairs
// that are counted fill the first warps, and the others have nothing to do.
template <int H>
struct Block {
    int p0, q0;    // first row tile, first column tile
    int rs;        // row slots of the tables; the columns' follow
    int count;     // its pairs (H 1)
    int r, c;      // this thread's pair, its first with H 2, as table slots
    bool diag;     // the column tiles are the row tiles
    // blk: of num_blocks(); first: the tiles below it have their pairs with one
    // another in the other launch
    __device__ __forceinline__ Block(int blk, int ntiles, int first) {
        const int tid = threadIdx.x;
        r = tid >> 4, c = tid & 15;
        if (H == 2) {
            const int n = first / 32, noff = n * (n - 1) / 2;
            // blocks off the diagonal first, then the cheaper diagonal ones
            int pb, qb;
            if (blk < noff)
                baseline_to_tiles(blk, n, pb, qb);
            else
                pb = qb = blk - noff;
            p0 = 32 * pb, q0 = 32 * qb, rs = 32, count = NTH;
            diag = pb == qb;
        } else {
            const int n = ntiles / 16, n0 = first / 16, noff = (n * (n - 1) - n0 * (n0 - 1)) / 2;
            int k = tid;
            rs = 16;
            diag = false;
            if (blk < noff) {
                const int x = blk + n0 * (n0 - 1) / 2;
                int qb = (int)((1.f + sqrtf(8.f * x + 1.f)) * 0.5f);
                while (qb * (qb - 1) / 2 > x) qb--;
                while (qb * (qb + 1) / 2 <= x) qb++;
                p0 = 16 * (x - qb * (qb - 1) / 2), q0 = 16 * qb;
                count = NTH;
            } else if (blk < noff + n - n0) {
                p0 = q0 = 16 * (n0 + blk - noff);
                count = 120;
                diag = true;
                baseline_to_tiles(k < count ? k : 0, 16, r, c);
            } else {
                q0 = 16 * n;
                const int nc = ntiles - q0;
                rs = GRP - nc;
                p0 = rs * (blk - noff - (n - n0));
                const int nr = min(rs, ntiles - p0), rect = min(max(q0 - p0, 0), nr);  // rows of other tiles
                const int i0 = max(p0 - q0, 0), i1 = p0 + nr - q0;                       // of the strip's own
                auto start = [&](int i) { return i * (2 * nc - i - 1) / 2; };
                count = rect * nc + (i1 > i0 ? start(i1) - start(i0) : 0);
                if (k >= count) k = 0;
                if (k < rect * nc) {
                    r = k / nc, c = k - r * nc;
                } else if (count > 0) {
                    baseline_to_tiles(k - rect * nc + start(i0), nc, r, c);
                    r += q0 - p0;
                } else {
                    r = c = 0;
                }
            }
        }
        c += rs;
    }
    // this thread has a pair (H 1)
    __device__ __forceinline__ bool mine() const { return (int)threadIdx.x < count; }
    // the tile of a table slot
    __device__ __forceinline__ int tile(int slot, int ntiles) const {
        const int t = slot < rs ? p0 + slot : q0 + slot - rs;
        return H == 2 ? min(t, ntiles - 1) : t;
    }
    // the visibility of a pair of table slots in channel f, or -1 (on or below
    // the diagonal, or past the array)
    __device__ __forceinline__ long long vis_index(const DirectParams& p, int f, int row, int col) const {
        const int tp = p0 + row, tq = q0 + col - rs;
        return tp < tq && tq < p.ntiles ? (long long)f * p.nbl + baseline_index(tp, tq, p.ntiles) : -1;
    }
};

// its blocks
static int num_blocks(int h, int ntiles, int first) {
    if (h == 2) return first / 32 * (first / 32 + 1) / 2;
    const int n = ntiles / 16, n0 = first / 16, rest = ntiles % 16;
    return (n * (n - 1) - n0 * (n0 - 1)) / 2 + n - n0 + (rest ? (ntiles + GRP - rest - 1) / (GRP - rest) : 0);
}

// vis[at[i]] += value(i) where at[i] is not negative.  Every load comes before
// the first store, so that the thread waits for them once (128 tiles x 384
// channels, one component: 92 us, a pair after another, 76 so).
template <bool OUT64, int N, class F>
__device__ __forceinline__ void add_pairs(void* vis, const long long (&at)[N], F&& value) {
    using V = typename std::conditional<OUT64, double2, float4>::type;
    constexpr int NV = OUT64 ? 4 : 2;
    V x[N][NV];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int e = 0; e < NV; e++)
            if (at[i] >= 0) x[i][e] = reinterpret_cast<const V*>(vis)[at[i] * NV + e];
#pragma unroll
    for (int i = 0; i < N; i++) {
        if (at[i] < 0) continue;
        const J2 d = value(i);
        const cplx c[4] = {d.a, d.b, d.c, d.d};
#pragma unroll
        for (int e = 0; e < NV; e++) {
            V y = x[i][e];
            if constexpr (OUT64) {
                y.x += c[e].re, y.y += c[e].im;
            } else {
                y.x += (float)c[2 * e].re, y.y += (float)c[2 * e].im;
                y.z += (float)c[2 * e + 1].re, y.w += (float)c[2 * e + 1].im;
            }
            reinterpret_cast<V*>(vis)[at[i] * NV + e] = y;
        }
    }
}

// Tile's UVW from the array's centroid in wavelengths (ool = frequency / c).
__device__ __forceinline__ void tile_uvw(const DirectParams& p, int tile, double ool, double& u, double& v, double& w) {
    const XYZ a = p.xyzs[tile];
    const double x = a.x - p.xyz0.x, y = a.y - p.xyz0.y, z = a.z - p.xyz0.z;
    u = (p.s_ha * x + p.c_ha * y) * ool;
    v = (-p.s_dec * p.c_ha * x + p.s_dec * p.s_ha * y + p.c_dec * z) * ool;
    w = (p.c_dec * p.c_ha * x - p.c_dec * p.s_ha * y + p.s_dec * z) * ool;
}

// 2^-x of x >= 0 (results below the smallest normal number become 0)
__device__ __forceinline__ float exp2_neg(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(-x));
    return r;
}

// components per staged chunk: what fits 48 KB of static shared memory with
// the per-tile tables
template <int TYPE, bool TILE>
struct Shape {
    static constexpr int CH = TILE ? 8 : (TYPE == 0 ? 32 : 16);
};

// Linear interpolation between the tabulated basis values around position
// pos (in table steps from the first entry), as sums over the dimensionless
// Hermite polynomials: out[n] = H_n(x0) e0 (1 - frac) + H_n(x1) e1 frac with
// x0, x1 the table's grid points and e = exp(-x^2 / 2); the factors
// 1 / sqrt(2^n n!) are folded into the coefficients.  Evaluating the two
// grid points (about 75 FP64 operations an axis) replaces twelve scattered
// 16-byte loads, which cost a warp some 380 L1 cycles.
__device__ __forceinline__ void hermite_interp(double pos, double (&out)[SDN]) {
    const double fl = floor(pos);
    const double frac = pos - fl;
    // positions outside the table take its first or last interval, where the
    // basis is zero
    const double k = fmin(fmax(fl, 0.0), (double)(SBF_L - 2));
    const double x0 = (k - SBF_C) * SBF_DX, x1 = (k + 1.0 - SBF_C) * SBF_DX;
    const double s0 = exp(-0.5 * (x0 * x0)) * (1.0 - frac), s1 = exp(-0.5 * (x1 * x1)) * frac;
    const double y0 = 2.0 * x0, y1 = 2.0 * x1;
    double a0 = s0, a1 = s1, b0 = y0 * s0, b1 = y1 * s1;  // H_n s of two consecutive orders
    out[0] = a0 + a1;
    out[1] = b0 + b1;
#pragma unroll
    for (int n = 2; n < SDN; n++) {
        const double c0 = fma(y0, b0, -2.0 * (n - 1) * a0), c1 = fma(y1, b1, -2.0 * (n - 1) * a1);
        a0 = b0, a1 = b1, b0 = c0, b1 = c1;
        out[n] = c0 + c1;
    }
}

// The shapelet envelope of table coordinates (dx, dy) from the table's
// centre with the component's signed dense coefficients cm [n1][n2].
__device__ __forceinline__ cplx shapelet_env(const double* __restrict__ cm, double dx, double dy) {
    double X[SDN], Y[SDN];
    hermite_interp(dx + SBF_C, X);
    hermite_interp(dy + SBF_C, Y);
    cplx e = {0.0, 0.0};
#pragma unroll
    for (int n1 = 0; n1 < SDN; n1++) {
        double tr = 0.0, ti = 0.0;
#pragma unroll
        for (int n2 = 0; n2 < SDN; n2++) {
            if ((n1 + n2) & 1)
                ti = fma(cm[n1 * SDN + n2], Y[n2], ti);
            else
                tr = fma(cm[n1 * SDN + n2], Y[n2], tr);
        }
        e.re = fma(X[n1], tr, e.re);
        e.im = fma(X[n1], ti, e.im);
    }
    return e;
}

// FAST (Gaussians): the envelope's exponential in FP32 of the FP64 base-2
// exponent (gp holds DirectParams::gk), as the chosen form takes it: rounding
// the exponent moves the envelope by ln2 |x| 6e-8 2^-|x| <= 2.2e-8 of the
// component's flux.  Only the chosen form with per-tile beams comes here, all
// else in FP64 (error's p99.9 3.4e-7 with FP32 phasors and left operands,
// 2.6e-7 so).  128 tiles x 192 channels x 250 Gaussians, 17 unique tiles: 2.37
// ms with a thread per baseline (phasors and records of 17 tiles gathered from
// shared memory per term), 1.84 so, the FP64 pipe 0.61 busy.
// H 1: three or, with per-tile beams, four CTAs an SM (65 tiles x 256 channels x
// 200 Gaussians: 881 us at three, 826 at four; points under a shared beam are
// slower by a tenth at four where the SMs are not full).
template <int TYPE, bool TILE, bool OUT64, bool FAST, int H>
__global__ void __launch_bounds__(NTH, H == 2 ? 2 : (TILE && TYPE != 2 ? 4 : 3)) pair_kernel(const DirectParams p, int first) {
    constexpr int CH = Shape<TYPE, TILE>::CH, SLOTS = H == 2 ? 64 : GRP;
    __shared__ alignas(128) double4 s_lmn[2][CH];
    __shared__ alignas(128) JonesF64 s_flux[2][CH];
    __shared__ alignas(128) double4 s_gp[TYPE ? 2 : 1][TYPE ? CH : 1];
    // shared beam: the phasors of the row tiles, then the column tiles;
    // per-tile beams: M_p and N_q entries (xx, xy, yx, yy)
    __shared__ alignas(16) double2 s_a[TILE ? 4 : 1][CH][SLOTS];
    __shared__ alignas(16) double2 s_k[TYPE ? CH : 1][TYPE ? SLOTS : 1];  // envelope coordinates
    __shared__ alignas(16) double4 s_w[TILE ? 1 : CH];                    // xx, yy, Re xy, Im xy
    __shared__ double s_dense[TYPE == 2 ? CH * SDN * SDN : 1];
    __shared__ alignas(8) uint64_t bar[2];

    // H 1: the channels are the faster index, so that CTAs of one cost are
    // spread over the SMs
    const int tid = threadIdx.x, f = H == 2 ? blockIdx.y : blockIdx.x % p.nf;
    const Block<H> B(H == 2 ? blockIdx.x : blockIdx.x / p.nf, p.ntiles, first);
    if (H == 1 && B.count == 0) return;
    const bool any = H == 2 || __any_sync(0xffffffffu, B.mine());

    // this thread's tile of the chunk tables: its UVW in wavelengths and, for
    // per-tile beams, its row of the beam table
    const int slot = tid & (SLOTS - 1), tile = B.tile(slot, p.ntiles);
    const double freq = p.freqs[f], ool = freq / VEL_C;
    double u = 0.0, v = 0.0, w = 0.0;
    const JonesF64* brow = nullptr;
    if (tile < p.ntiles) {
        tile_uvw(p, tile, ool, u, v, w);
        if (TILE) brow = p.beam + (size_t)p.nc * ((size_t)p.n_uniq_freq * p.tile_map[tile] + p.freq_map[f]);
    }

    // a diagonal block's column tiles are its row tiles: formed once (per-tile
    // beams need both M and N)
    const bool same = !TILE && B.diag;

    // H 2, a diagonal block: its two diagonal quarters hold half as many pairs
    // each and are one quarter's work, pair 0, of which the threads below the
    // diagonal take the mirrored pair of the second; pair 1 is the full quarter's
    const bool mirror = H == 2 && B.diag && B.r > B.c - 32;
    const int r00 = mirror ? 16 + B.c - 32 : B.r, c00 = mirror ? 48 + B.r : B.c;

    const int nchunks = (p.nc + CH - 1) / CH;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();
    auto issue = [&](int k) {
        const int st = k & 1, c0 = k * CH, n = min(CH, p.nc - c0);
        mbar_arrive_expect_tx(&bar[st], n * 32u + n * 64u + (TYPE ? n * 32u : 0u));
        bulk_g2s(s_lmn[st], p.lmn + c0, n * 32u, &bar[st]);
        bulk_g2s(s_flux[st], p.flux + (size_t)f * p.nc + c0, n * 64u, &bar[st]);
        if (TYPE) bulk_g2s(s_gp[st], p.gp + c0, n * 32u, &bar[st]);
    };
    int issued = 0;  // chunks whose copies thread 0 has issued
    if (tid == 0) {
        fence_proxy_async_smem();
        if (!p.stall) {
            if (nchunks > 0) issue(0), issued = 1;
            if (nchunks > 1) issue(1), issued = 2;
        }
    }
    const uint64_t limit = p.wait_ns ? p.wait_ns : 2000000000ull;

    // shared beam: sums of w_xx z, w_yy z, Re(w_xy) z, Im(w_xy) z; per-tile
    // beams: the four correlations
    cplx acc[H * H][4];
#pragma unroll
    for (int i = 0; i < H * H; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][e] = cplx{0.0, 0.0};

    bool aborted = false;
    for (int k = 0; k < nchunks; k++) {
        const int st = k & 1;
        const bool ok = mbar_wait_bounded(&bar[st], (k >> 1) & 1, p.err, limit);
        const int c0 = k * CH, n = ok ? min(CH, p.nc - c0) : 0;

        // ---- the chunk's per-tile tables ----
        if (tile < p.ntiles && (!same || slot < SLOTS / 2)) {
            for (int c = tid / SLOTS; c < n; c += NTH / SLOTS) {
                const double4 lmn = s_lmn[st][c];
                const cplx a = phasor_quarter_f64(4.0 * (u * lmn.x + v * lmn.y + w * lmn.z));
                if (!TILE) {
                    const double2 x = make_double2(a.re, a.im);
                    s_a[0][c][slot] = x;
                    if (same) s_a[0][c][slot + SLOTS / 2] = x;
                } else {
                    J2 b = ldg_j(brow + c0 + c);
                    if (slot < B.rs) b = b * load_j(s_flux[st][c]);
                    b = b * a;
                    s_a[0][c][slot] = make_double2(b.a.re, b.a.im);
                    s_a[TILE ? 1 : 0][c][slot] = make_double2(b.b.re, b.b.im);
                    s_a[TILE ? 2 : 0][c][slot] = make_double2(b.c.re, b.c.im);
                    s_a[TILE ? 3 : 0][c][slot] = make_double2(b.d.re, b.d.im);
                }
                if (TYPE) {
                    const double4 g = s_gp[TYPE ? st : 0][TYPE ? c : 0];
                    double2 x;
                    if (TYPE == 1) {
                        x = FAST ? make_double2(u * g.x + v * g.y, u * g.z + v * g.w)
                                 : make_double2(u * g.z + v * g.w, u * g.w - v * g.z);
                    } else {
                        const double2 q = __ldg(p.suv_tile + (size_t)(c0 + c) * p.ntiles + tile);
                        const double su = q.x * ool, sv = q.y * ool;
                        x = make_double2((su * g.z + sv * g.w) * g.x, (su * g.w - sv * g.z) * g.y);
                    }
                    s_k[TYPE ? c : 0][TYPE ? slot : 0] = x;
                    if (same) s_k[TYPE ? c : 0][TYPE ? slot + SLOTS / 2 : 0] = x;
                }
            }
        }
        if (!TILE && tid < n) {
            const JonesF64 q = s_flux[st][tid];
            s_w[TILE ? 0 : tid] = make_double4(q.j00_re, q.j11_re, q.j01_re, q.j01_im);
        }
        if (TYPE == 2)
            for (int i = tid; i < n * SDN * SDN; i += NTH) s_dense[TYPE == 2 ? i : 0] = __ldg(p.sdense64 + (size_t)c0 * SDN * SDN + i);
        if (__syncthreads_or(!ok)) {
            // the sum is incomplete: leave the visibilities untouched
            if (tid == 0) drain_two_stage(bar, k, issued);
            aborted = true;
            break;
        }

        // ---- the pairs ----
        auto term = [&](int c, int i, int rp, int cq) {
            cplx env = {1.0, 0.0};
            if (TYPE) {
                const double2 kp = s_k[TYPE ? c : 0][TYPE ? rp : 0], kq = s_k[TYPE ? c : 0][TYPE ? cq : 0];
                const double dx = kp.x - kq.x, dy = kp.y - kq.y;
                if (TYPE == 1 && FAST) {
                    env.re = (double)exp2_neg((float)fma(dx, dx, dy * dy));
                } else if (TYPE == 1) {
                    const double4 g = s_gp[TYPE ? st : 0][TYPE ? c : 0];
                    env.re = exp(g.x * (dx * dx) + g.y * (dy * dy));
                } else {
                    env = shapelet_env(s_dense + (TYPE == 2 ? c * SDN * SDN : 0), dx, dy);
                }
            }
            cplx(&m)[4] = acc[i];
            if (!TILE) {
                const double2 ap = s_a[0][c][rp], aq = s_a[0][c][cq];
                cplx z = {fma(ap.x, aq.x, ap.y * aq.y), fma(ap.y, aq.x, -(ap.x * aq.y))};
                if (TYPE == 1) z = z * env.re;
                if (TYPE == 2) z = z * env;
                const double4 wv = s_w[TILE ? 0 : c];
                const double we[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    m[e].re = fma(we[e], z.re, m[e].re);
                    m[e].im = fma(we[e], z.im, m[e].im);
                }
            } else {
                cplx M[4], N[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const double2 a = s_a[TILE ? e : 0][c][rp], b = s_a[TILE ? e : 0][c][cq];
                    M[e] = cplx{a.x, a.y};
                    N[e] = cplx{b.x, b.y};
                    if (TYPE == 1) M[e] = M[e] * env.re;
                    if (TYPE == 2) M[e] = M[e] * env;
                }
#pragma unroll
                for (int a = 0; a < 2; a++)
#pragma unroll
                    for (int b = 0; b < 2; b++)
#pragma unroll
                        for (int y = 0; y < 2; y++) {
                            // M^{ay} conj(N^{by})
                            const cplx x = M[2 * a + y], q = N[2 * b + y];
                            cplx& o = m[2 * a + b];
                            o.re = fma(x.re, q.re, fma(x.im, q.im, o.re));
                            o.im = fma(x.im, q.re, fma(-x.re, q.im, o.im));
                        }
            }
        };
        if (H == 1) {
            for (int c = 0; c < n && any; c++) term(c, 0, B.r, B.c);
        } else if (!B.diag) {
            for (int c = 0; c < n; c++)
#pragma unroll
                for (int i = 0; i < H * H; i++) term(c, i, B.r + 16 * (i / H), B.c + 16 * (i % H));
        } else {
            for (int c = 0; c < n; c++) {
                term(c, 0, r00, c00);
                term(c, H - 1, B.r, B.c + 16);
            }
        }
        __syncthreads();
        if (tid == 0 && k + 2 < nchunks) {
            fence_proxy_async_smem();
            issue(k + 2);
            issued = k + 3;
        }
    }

    if (aborted || (H == 1 && !B.mine())) return;
    long long at[H * H];
#pragma unroll
    for (int i = 0; i < H * H; i++) {
        const int rp = H == 2 && i == 0 ? r00 : B.r + 16 * (i / H), cq = H == 2 && i == 0 ? c00 : B.c + 16 * (i % H);
        at[i] = H == 2 && B.diag && i > 1 ? -1 : B.vis_index(p, f, rp, cq);
    }
    add_pairs<OUT64>(p.vis, at, [&](int i) {
        const cplx(&m)[4] = acc[i];
        if (TILE) return J2{m[0], m[1], m[2], m[3]};
        return J2{m[0], cplx{m[2].re - m[3].im, m[2].im + m[3].re}, cplx{m[2].re + m[3].im, m[2].im - m[3].re}, m[1]};
    });
}

// The tiles (a multiple of 32, or past the array) whose pairs with one another
// go in blocks of 32 x 32; 0: none.  Those blocks reuse what they read from
// shared memory, but a CTA's work is four times as much, so that they need
// enough of them for each SM: twice as many for FP64 Gaussians, whose
// exponentials are bound by the FP64 pipe either way, fewer for the points.  60
// components, us in 32 x 32 / 16 x 16 blocks, 128 tiles:
//                          24 channels  64         128        384
//   points                 39 / 39      66 / 74    104 / 123  259 / 324
//   Gaussians              75 / 68      141 / 141  242 / 258  645 / 716
//   Gaussians, chosen form 41 / 41      71 / 78    115 / 140  300 / 370
//   same, per-tile beams   128 / 119    224 / 222  359 / 381  932 / 1037
// (2534 points, 151 tiles x 28 channels: 1241 / 1388.)  A last group of fewer
// than 23 tiles goes in strips of the other launch, which pays later (111 tiles
// x 128 channels, points: 100 / 103, Gaussians of the chosen form 118 / 116, with
// per-tile beams 350 / 330); one of 23 or more is padded (123 tiles x 128
// channels, points: 105 padded, 121 with strips).
// Shapelets evaluate their basis per pair and take 16 x 16 blocks at any size
// (128 tiles x 384 channels x 20: 1097 / 1010 us).
static int whole_tiles(const DirectParams& p, int type, bool tile_beam, bool fast) {
    if (type == 2) return 0;
    const int n = (p.ntiles + 9) / 32;
    const bool strips = 32 * n < p.ntiles;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    double ctas;  // blocks of 32 x 32 per SM from which they pay
    if (type == 1 && !fast)
        ctas = 8.0;
    else if (tile_beam)
        ctas = strips ? 6.0 : 4.0;
    else
        ctas = type == 0 && !strips ? 2.5 : 4.0;
    return 0.5 * n * (n + 1) * p.nf >= ctas * sms ? 32 * n : 0;
}

template <int H>
static dim3 block_grid(const DirectParams& p, int first) {
    const int n = num_blocks(H, p.ntiles, first);
    return H == 2 ? dim3(n, p.nf) : dim3(n * p.nf);
}

template <int TYPE, bool TILE, bool FAST, int H>
cudaError_t launch_h(bool out64, const DirectParams& p, int first, cudaStream_t s) {
    const dim3 grid = block_grid<H>(p, first);
    if (out64)
        pair_kernel<TYPE, TILE, true, FAST, H><<<grid, NTH, 0, s>>>(p, first);
    else
        pair_kernel<TYPE, TILE, false, FAST, H><<<grid, NTH, 0, s>>>(p, first);
    count_launches(1);
    return cudaGetLastError();
}

template <int TYPE, bool TILE, bool FAST = false>
cudaError_t launch_t(bool out64, const DirectParams& p, cudaStream_t s) {
    const int first = whole_tiles(p, TYPE, TILE, FAST);
    if constexpr (TYPE != 2) {
        const cudaError_t e = first ? launch_h<TYPE, TILE, FAST, 2>(out64, p, first, s) : cudaSuccess;
        if (e != cudaSuccess) return e;
    }
    return first < p.ntiles ? launch_h<TYPE, TILE, FAST, 1>(out64, p, first, s) : cudaSuccess;
}

}  // namespace pairs

cudaError_t launch_pairs(int ty, bool tile_beam, bool out64, const DirectParams& p, cudaStream_t s) {
    if (ty == 0)
        return tile_beam ? pairs::launch_t<0, true>(out64, p, s) : pairs::launch_t<0, false>(out64, p, s);
    if (ty == 1)
        return tile_beam ? pairs::launch_t<1, true>(out64, p, s) : pairs::launch_t<1, false>(out64, p, s);
    return tile_beam ? pairs::launch_t<2, true>(out64, p, s) : pairs::launch_t<2, false>(out64, p, s);
}

// ---------------------------------------------------------------------------
// The chosen (tensor) form's Gaussians with a shared beam, factored by tile
// as above: FP32 phasors per tile after the FP64 phase and its exact range
// reduction; the envelope's base-2 exponent -|K_p - K_q|^2 from FP64 per-tile
// coordinates K held as two FP32 numbers (a multiple of 2^-8, whose
// differences and squares are exact where the envelope is not zero, and the
// rest), rounded once per axis; products and sums over SUM chunks in FP32,
// those sums in FP64 (kept in shared memory between, so that a thread's
// registers hold only the FP32 ones).  Products are packed in pairs
// (fma.rn.f32x2: two FP32 operations an issue slot).
//
// Bound: shared-memory reads (128 bytes a clock and SM, whether or not lanes
// share an address: 28 bytes a lane and term here) and the issue slots, about
// 24 warp instructions a term (a thread per baseline, with the phasor per
// baseline and unpacked: 64).  500 Gaussians, 128 tiles x 384 channels: 2.75
// ms -> 2.08 ms; with an FP64 exponent per pair and packed phasors stored
// ready 2.39 ms (40 bytes a lane and term); 4 x 2 pairs at half the warps
// 2.38 ms.
// ---------------------------------------------------------------------------
namespace pairs {

constexpr int FCHUNK = 16;  // components per staged chunk
constexpr int SUM = 2;      // chunks summed in FP32

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// An FP64 coordinate's upper part: x rounded to a multiple of 2^-8 (|x| < 2^14, else to FP32)
__device__ __forceinline__ float coarse(double x) {
    const float f = (float)x;
    constexpr float M = 49152.f;
    return fabsf(f) < 16384.f ? __fsub_rn(__fadd_rn(f, M), M) : f;
}

template <int H>
struct FastSmem {
    static constexpr int SLOTS = H == 2 ? 64 : GRP;
    double4 lmn[2][FCHUNK];
    JonesF64 flux[2][FCHUNK];
    double4 gp[2][FCHUNK];     // K = (u gp.x + v gp.y, u gp.z + v gp.w): the exponent is -|K_p - K_q|^2
    float2 a[FCHUNK][SLOTS];  // phasors of the row tiles, then the column tiles
    float4 k[FCHUNK][SLOTS];  // envelope coordinates (hx, hy, lx, ly), negated for column tiles
    float4 w[FCHUNK];         // xx, yy, Re xy, Im xy
    double2 sum[H * H][4][NTH];  // [pair][sum][thread]
    uint64_t bar[2];
};

template <bool OUT64, int H>
__global__ void __launch_bounds__(NTH, H == 2 ? 2 : 4) fast_gauss_kernel(const DirectParams p, int first) {
    constexpr int SLOTS = FastSmem<H>::SLOTS;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FastSmem<H>& S = *reinterpret_cast<FastSmem<H>*>(smem_raw);
    const int tid = threadIdx.x, f = H == 2 ? blockIdx.y : blockIdx.x % p.nf;
    const Block<H> B(H == 2 ? blockIdx.x : blockIdx.x / p.nf, p.ntiles, first);
    if (H == 1 && B.count == 0) return;
    // warps without a pair have nothing to sum
    const bool any = H == 2 || __any_sync(0xffffffffu, B.mine());

    const int slot = tid & (SLOTS - 1), tile = B.tile(slot, p.ntiles);
    const double freq = p.freqs[f], ool = freq / VEL_C;
    double u = 0.0, v = 0.0, w = 0.0;  // wavelengths
    if (tile < p.ntiles) tile_uvw(p, tile, ool, u, v, w);
    const int rp = B.r, cq = B.c;

    const int nchunks = (p.nc + FCHUNK - 1) / FCHUNK;
    if (tid == 0) {
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();
    auto issue = [&](int k) {
        const int st = k & 1, c0 = k * FCHUNK, n = min(FCHUNK, p.nc - c0);
        mbar_arrive_expect_tx(&S.bar[st], n * 128u);
        bulk_g2s(S.lmn[st], p.lmn + c0, n * 32u, &S.bar[st]);
        bulk_g2s(S.flux[st], p.flux + (size_t)f * p.nc + c0, n * 64u, &S.bar[st]);
        bulk_g2s(S.gp[st], p.gk + c0, n * 32u, &S.bar[st]);
    };
    int issued = 0;  // chunks whose copies thread 0 has issued
    if (tid == 0) {
        fence_proxy_async_smem();
        if (!p.stall) {
            if (nchunks > 0) issue(0), issued = 1;
            if (nchunks > 1) issue(1), issued = 2;
        }
    }
    const uint64_t limit = p.wait_ns ? p.wait_ns : 2000000000ull;

    uint64_t acc[H * H][4];  // [pair] (re, im) of the sums of w_xx z, w_yy z, Re(w_xy) z, Im(w_xy) z
#pragma unroll
    for (int i = 0; i < H * H; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][e] = 0;

    const uint64_t two = dup2(2.f);
    bool aborted = false;
    for (int k = 0; k < nchunks; k++) {
        const int st = k & 1;
        const bool ok = mbar_wait_bounded(&S.bar[st], (k >> 1) & 1, p.err, limit);
        const int n = ok ? min(FCHUNK, p.nc - k * FCHUNK) : 0;
        if (tid < n) {
            const JonesF64 q = S.flux[st][tid];
            S.w[tid] = make_float4((float)q.j00_re, (float)q.j11_re, (float)q.j01_re, (float)q.j01_im);
        }
        if (tile < p.ntiles && (!B.diag || slot < SLOTS / 2)) {
            for (int c = tid / SLOTS; c < n; c += NTH / SLOTS) {
                const double4 lmn = S.lmn[st][c], sc = S.gp[st][c];
                float sn, cs;
                phasor_quarter_f32(4.0 * (u * lmn.x + v * lmn.y + w * lmn.z), sn, cs);
                const double2 xx = make_double2(u * sc.x + v * sc.y, u * sc.z + v * sc.w);
                const float hx = coarse(xx.x), hy = coarse(xx.y);
                const float4 x = make_float4(hx, hy, (float)(xx.x - (double)hx), (float)(xx.y - (double)hy));
                const float4 nx = make_float4(-x.x, -x.y, -x.z, -x.w);
                S.a[c][slot] = make_float2(cs, sn);
                S.k[c][slot] = slot < B.rs ? x : nx;
                if (B.diag) {
                    S.a[c][slot + SLOTS / 2] = make_float2(cs, sn);
                    S.k[c][slot + SLOTS / 2] = nx;
                }
            }
        }
        if (__syncthreads_or(!ok)) {
            // the sum is incomplete: leave the visibilities untouched
            if (tid == 0) drain_two_stage(S.bar, k, issued);
            aborted = true;
            break;
        }

        // in stages over the thread's pairs, so that their chains (loads,
        // exponent, exponential) overlap; a pair that is no baseline (H 2: below
        // the diagonal in a quarter on it; H 1: past the count in a warp that
        // holds some) is summed like the others and not stored
        auto sweep = [&](auto diag) {
            constexpr bool DIAG = decltype(diag)::value;  // the lower left quarter holds no baseline
            for (int c = 0; c < n; c++) {
                const ulonglong2* kr = reinterpret_cast<const ulonglong2*>(S.k[c]);
                ulonglong2 kq[H];
#pragma unroll
                for (int j = 0; j < H; j++) kq[j] = kr[cq + 16 * j];
                float e[H * H];
#pragma unroll
                for (int i = 0; i < H; i++) {
                    const ulonglong2 kp = kr[rp + 16 * i];
#pragma unroll
                    for (int j = 0; j < H; j++) {
                        if (DIAG && i > j) continue;
                        // dh^2 + dl (2 dh + dl): dh exact, one rounding
                        const uint64_t dh = add2(kp.x, kq[j].x), dl = add2(kp.y, kq[j].y);
                        const float2 q = unpack2(fma2(dh, dh, mul2(dl, fma2(two, dh, dl))));
                        e[H * i + j] = q.x + q.y;
                    }
                }
                const float4 wv = S.w[c];
                const uint64_t w[4] = {dup2(wv.x), dup2(wv.y), dup2(wv.z), dup2(wv.w)};
                uint64_t qx[H], qy[H];
#pragma unroll
                for (int j = 0; j < H; j++) {
                    const float2 aq = S.a[c][cq + 16 * j];
                    qx[j] = dup2(aq.x);
                    qy[j] = dup2(aq.y);
                }
#pragma unroll
                for (int i = 0; i < H; i++) {
                    const float2 ap = S.a[c][rp + 16 * i];
                    const uint64_t px = pack2(ap.x, ap.y), py = pack2(ap.y, -ap.x);
#pragma unroll
                    for (int j = 0; j < H; j++) {
                        if (DIAG && i > j) continue;
                        uint64_t(&m)[4] = acc[H * i + j];
                        const uint64_t z = mul2(fma2(py, qy[j], mul2(px, qx[j])), dup2(exp2_neg(e[H * i + j])));
#pragma unroll
                        for (int x = 0; x < 4; x++) m[x] = fma2(w[x], z, m[x]);
                    }
                }
            }
        };
        if (H == 2 && B.diag)
            sweep(std::true_type{});
        else if (any)
            sweep(std::false_type{});
        if (k % SUM == SUM - 1 || k == nchunks - 1) {
            const bool first = k < SUM;
#pragma unroll
            for (int i = 0; i < H * H; i++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float2 a = unpack2(acc[i][e]);
                    double2 s = first ? make_double2(0.0, 0.0) : S.sum[i][e][tid];
                    s.x += (double)a.x;
                    s.y += (double)a.y;
                    S.sum[i][e][tid] = s;
                    acc[i][e] = 0;
                }
        }
        __syncthreads();
        if (tid == 0 && k + 2 < nchunks) {
            fence_proxy_async_smem();
            issue(k + 2);
            issued = k + 3;
        }
    }

    if (aborted || (H == 1 && !B.mine())) return;
    long long at[H * H];
#pragma unroll
    for (int i = 0; i < H * H; i++) at[i] = B.vis_index(p, f, rp + 16 * (i / H), cq + 16 * (i % H));
    add_pairs<OUT64>(p.vis, at, [&](int i) {
        const double2 xx = S.sum[i][0][tid], yy = S.sum[i][1][tid], a = S.sum[i][2][tid], b = S.sum[i][3][tid];
        return J2{{xx.x, xx.y}, {a.x - b.y, a.y + b.x}, {a.x + b.y, a.y - b.x}, {yy.x, yy.y}};
    });
}

template <bool OUT64, int H>
cudaError_t launch_fast_gauss(const DirectParams& p, int first, cudaStream_t s) {
    // the opt-in above 48 KB of dynamic shared memory, once per device
    static std::atomic<bool> attr[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr[dev].load(std::memory_order_relaxed)) {
        e = cudaFuncSetAttribute(fast_gauss_kernel<OUT64, H>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(FastSmem<H>));
        if (e != cudaSuccess) return e;
        attr[dev].store(true, std::memory_order_relaxed);
    }
    fast_gauss_kernel<OUT64, H><<<block_grid<H>(p, first), NTH, sizeof(FastSmem<H>), s>>>(p, first);
    count_launches(1);
    return cudaGetLastError();
}

template <bool OUT64>
cudaError_t launch_fast_gauss(const DirectParams& p, cudaStream_t s) {
    const int first = whole_tiles(p, 1, false, true);
    const cudaError_t e = first ? launch_fast_gauss<OUT64, 2>(p, first, s) : cudaSuccess;
    return e != cudaSuccess || first >= p.ntiles ? e : launch_fast_gauss<OUT64, 1>(p, first, s);
}

}  // namespace pairs

cudaError_t launch_fast_gauss(bool tile_beam, bool out64, const DirectParams& p, cudaStream_t s) {
    if (tile_beam) {
        DirectParams q = p;
        q.gp = p.gk;
        return pairs::launch_t<1, true, true>(out64, q, s);
    }
    return out64 ? pairs::launch_fast_gauss<true>(p, s) : pairs::launch_fast_gauss<false>(p, s);
}

}  // namespace hdc

// Direct FP64 predictor kernels (shared by the drop-in entry points and the
// native modeller).
#pragma once

#include "common.cuh"

namespace hdc {

// Per-type component tables consumed by the direct kernel.  Component order
// is the modelling order; for the drop-in layer it is power laws, curved
// power laws, lists (gpu/types.h:187-267), which is also the beam-direction
// order of d_beam_jones.
constexpr int SDN = SDN_TABLE;  // orders 0..5 in the dense shapelet form

struct DirectParams {
    int nbl, nf, ntiles, nc;
    const double* freqs;  // [nf] Hz
    const UVW* uvws;      // [nbl] m
    const double4* lmn;   // [nc] (l, m, n - 1, 0), dimensionless (turn units)
    const JonesF64* flux; // [nf][nc]: B S B^H when the beam is shared (or none), S when per tile
    const double4* gp;    // [nc] Gaussian: (C maj^2, C min^2, sin pa, cos pa); shapelet: (maj K, -min K, sin pa, cos pa)
    const double4* gk;    // [nc] Gaussians of the chosen form: rows of the 2 x 2 matrix that takes (u, v) to the
                          // coordinates whose squared length is the envelope's base-2 exponent, or NULL
    // per-tile beam, reference layout [uniq_tile][uniq_freq][nc]
    const JonesF64* beam;
    const int* tile_map;
    const int* unflagged_map;
    const int* freq_map;
    int n_uniq_freq;
    int n_uniq_tile;  // rows of beam (the chosen form's per-tile kernel stages them; 0: not known)
    // shapelets
    const double* sbf;  // [SBF_N][SBF_L]
    const float* sbf32; // the same table in FP32 (chosen form), or NULL
    // chosen form, orders below SDN: the table in FP32, position-major
    // [SBF_L][SDN / 2] float4, each (v, v', d, d') of two neighbouring orders
    // with v the value at the position and d the next position's less v; and
    // per component a dense SDN x SDN coefficient matrix [nc][n1][n2] with the
    // sign of i^(n1+n2) folded in; NULL when some coefficient's order is SDN or
    // more
    const float4* sbfp;
    const float* sdense;
    const ShapeletCoeff* coeffs;
    const int* coeff_start;
    const int* coeff_count;
    const ShapeletUV* suv_bl;  // [nbl][nc] m, or NULL
    const double2* suv_tile;   // [nc][ntiles] m, or NULL (then suv = tile1 - tile2)
    // the native modeller's tiles, when the UVWs are their differences (the
    // FP64 form factored by tile): geodetic positions and their centroid, and
    // the phase centre's hour angle and declination; NULL otherwise
    const XYZ* xyzs;
    XYZ xyz0;
    double s_ha, c_ha, s_dec, c_dec;
    // the dense coefficients for that form: FP64, with the basis functions'
    // normalisation folded in, or NULL
    const double* sdense64;
    void* vis;                 // [nf][nbl] JonesF32 or JonesF64, accumulated
    int* err;
    // Limit of each bounded wait on the staged tables [ns] (0: the default
    // 2 s).  stall != 0 (set only through hdc_test_stall_next_predict) issues
    // none of the table copies, so that the first wait runs out with nothing
    // in flight.
    unsigned long long wait_ns;
    int stall;
};

// Static message for a kernel error word (KERR_* bits), NULL for 0.
const char* kernel_error_string(int word);
// Status code of a kernel error word for the native layer (HDC_OK for 0).
int kernel_error_status(int word);

// vis[o] += acc (JonesF64 or JonesF32 [channel][baseline] at element o).
template <bool OUT64>
__device__ __forceinline__ void add_vis(void* vis, size_t o, const J2& acc) {
    if (OUT64) {
        double2* q = reinterpret_cast<double2*>(reinterpret_cast<JonesF64*>(vis) + o);
        const double2 a0 = q[0], b0 = q[1], c0 = q[2], d0 = q[3];
        q[0] = make_double2(a0.x + acc.a.re, a0.y + acc.a.im);
        q[1] = make_double2(b0.x + acc.b.re, b0.y + acc.b.im);
        q[2] = make_double2(c0.x + acc.c.re, c0.y + acc.c.im);
        q[3] = make_double2(d0.x + acc.d.re, d0.y + acc.d.im);
    } else {
        float4* q = reinterpret_cast<float4*>(reinterpret_cast<JonesF32*>(vis) + o);
        float4 x = q[0], y = q[1];
        x.x += (float)acc.a.re;
        x.y += (float)acc.a.im;
        x.z += (float)acc.b.re;
        x.w += (float)acc.b.im;
        y.x += (float)acc.c.re;
        y.y += (float)acc.c.im;
        y.z += (float)acc.d.re;
        y.w += (float)acc.d.im;
        q[0] = x;
        q[1] = y;
    }
}

// The FP64 predict of component type ty factored by tile (pairs.cu); p.xyzs
// set, shapelets with p.sdense64.
cudaError_t launch_pairs(int ty, bool tile_beam, bool out64, const DirectParams& p, cudaStream_t s);
// The chosen form's Gaussians factored by tile (a shared beam in FP32, a beam
// per tile with FP64 products); p.xyzs and p.gk set.
cudaError_t launch_fast_gauss(bool tile_beam, bool out64, const DirectParams& p, cudaStream_t s);

// Predict component type ty (0 point, 1 Gaussian, 2 shapelet) with the kernel
// that its geometry and beam allow.  tile_beam selects per-tile beam Jones;
// out64 an FP64 output; fast the chosen form's Gaussians and shapelets (errors
// ~1e-7 of the visibility).
cudaError_t launch_direct(int ty, bool tile_beam, bool out64, const DirectParams& p, cudaStream_t s,
                          bool fast = false);

// components of a TensorBeam::beam32 row (pairs are read in one aligned load)
__host__ __device__ inline size_t beam32_row(int nc) { return ((size_t)nc + 1) & ~(size_t)1; }

// Per-tile beams for the tensor-core predict: beam [n_uniq_tile]
// [n_uniq_freq][nc] (the reference's layout), the unique row of every tile
// (any unflagged-tile map already applied) and the unique column of every
// channel of the launch.
struct TensorBeam {
    const JonesF64* beam;
    const float4* beam32;  // its rows in FP32 (the producers' reads), or NULL: [unique tile][unique
                           // frequency][row X, Y][beam32_row(nc)], a row entry as re, im of its two columns
    const int* tile_map;
    const int* freq_map;
    int n_uniq_tile;
    int n_uniq_freq;
};

// A second stream and its events, with which the tensor predict writes the
// next chunk's table while the Gram kernel of the current chunk runs (two tables in the workspace).  One per caller: not shared
// between concurrent calls.
struct TensorSync {
    cudaStream_t ts = nullptr;
    cudaEvent_t start = nullptr, table_done[2] = {nullptr, nullptr}, gram_done[2] = {nullptr, nullptr};
};
int tensor_sync_init(TensorSync& t);
void tensor_sync_free(TensorSync& t);

// The tensor-core point predict of one timestep (csrc/tensor.cu): d_W is
// B S B^H [nf][nc] with a beam shared by all tiles (beam NULL), or S [nf][nc]
// with per-tile beams.  ws: ws_bytes >= tensor_workspace_bytes(nf, nbl,
// ntiles, nc, unique tiles of per-tile beams or 0, out64, sync != NULL, least)
// bytes; least takes per-tile beams' table of one channel at a time.  sync
// NULL runs every kernel on s in turn.
size_t tensor_workspace_bytes(int nf, int nbl, int ntiles, int nc, int n_uniq_tile, bool out64, bool two_tables,
                              bool least);
// Per-chunk output of the table form (shared beam, nc <= tensor_single_pass()
// components, JonesF32 output): after the Gram products of channels
// [f0, f0 + nch) the chunk's visibilities become vis + model + planes (model:
// [nf][nbl], added before the planes), and done(ctx, f0, nch) is called to
// queue the chunk's further work on s; no whole-array combine follows.
struct TensorChunkOut {
    const JonesF32* model;
    int (*done)(void* ctx, int f0, int nch);
    void* ctx;
};
int tensor_single_pass();
int launch_tensor_points(int nf, int nbl, int ntiles, int nc, const double* d_freqs, const XYZ* d_xyzs, double ha,
                         double dec, const double4* d_lmn, const JonesF64* d_W, const TensorBeam* beam, void* d_vis,
                         bool out64, void* ws, size_t ws_bytes, int* d_err, cudaStream_t s, TensorSync* sync,
                         const TensorChunkOut* chunk_out = nullptr);

struct AutosParams {
    int ntiles, nf;
    int nc_total;
    // up to 3 type tables concatenated by the caller into one [nf][nc] flux
    // table (S) and a beam table [uniq_tile][uniq_freq][nc] (NULL: identity)
    const JonesF64* flux;
    const JonesF64* beam;
    const int* tile_map;
    const int* unflagged_map;
    const int* freq_map;
    int n_uniq_freq;
    int n_uniq_tile;  // rows of beam (the chosen form's per-tile kernel stages them; 0: not known)
    JonesF32* vis;  // [nf][ntiles]
};
cudaError_t launch_autos(const AutosParams& p, cudaStream_t s);

// mask_pols over a [n] JonesF32 buffer (model/mod.rs:264-285)
cudaError_t launch_mask_pols(JonesF32* vis, size_t n, int pols, cudaStream_t s);

}  // namespace hdc

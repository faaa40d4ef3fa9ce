// What the two peel loops share (host side).
#pragma once

#include "modeller.cuh"

namespace hdc {

// call-scoped device buffers from the library's stream-ordered pool: freed
// blocks stay mapped, so later calls reuse them without new mappings
struct DevBuf {
    void* p = nullptr;
    cudaStream_t s = nullptr;
    bool pooled = false;
    cudaError_t alloc(size_t bytes, cudaStream_t st) {
        s = st;
        pooled = true;
        return pool_malloc_async(&p, bytes, st);
    }
    // large one-off buffers stay outside the pool, which keeps what it holds
    cudaError_t alloc_plain(size_t bytes) { return device_malloc(&p, bytes); }
    ~DevBuf() {
        if (p) pooled ? cudaFreeAsync(p, s) : cudaFree(p);
    }
    template <class T>
    T* as() {
        return reinterpret_cast<T*>(p);
    }
};

// Device state of one source's fit.
struct IonoDev {
    double alpha, beta, gain;
    int stop;
    int pad;  // blocks of the current iteration that have finished (iono_traces_kernel)
};

cudaError_t k_xyzs_to_uvws(const XYZ* xyzs, const double* lmsts, UVW* uvws, RADec pc, int ntiles, int nbl, int nt,
                           cudaStream_t s);
cudaError_t k_weights_average(const float* w, float* lo, int nt, int nbl, int nf, int favg, cudaStream_t s);
cudaError_t k_rotate(JonesF32* vis, int nt, int nbl, int nf, const UVW* from, const UVW* to, const double* lambdas,
                     cudaStream_t s);

// The fits of a batch of sources from the traces (XX + YY) of their
// low-resolution data and models, on one stream, nothing read back: states
// [nsrc] at (0, 0, 1) in and out, partials from iono_partials_bytes; then the
// constants neu = old + fit, or old where the reference's rule reverts them
// (|alpha| or |beta| > 1e-3, gain < 0 or > 1.5; gpu.rs:541-627).
size_t iono_partials_bytes(int nsrc, int nbl);
cudaError_t iono_states_init(IonoDev* states, int nsrc, cudaStream_t s);
cudaError_t iono_fit(const float2* d_resid, const float* d_w, const float2* d_model, double* d_partials,
                     IonoDev* d_states, const IonoConsts* d_old, IonoConsts* d_neu, int nsrc, int nbl, int nf, int niter,
                     const UVW* d_uvws, const double* d_lambdas, double convergence, cudaStream_t s);

// The source-by-source loop's two passes over the residual (peel.cu).
struct SeqArgs {
    JonesF32* resid;        // [nt][nf][nbl], in the frame of `from`
    const float* w;         // [nt][nf][nbl]
    const JonesF32* model;  // [nt][nf][nbl] in the source's frame, or NULL:
    const float4* point;    // [nt][nf] (xx, yy, Re xy, Im xy), the same on every baseline
    const IonoConsts *old, *neu;
    const UVW *from, *to;   // [nt][nbl]
    const double* lam;      // [nf] lambda
    int nt, nf, nbl, favg;
};
cudaError_t seq_accumulate(const SeqArgs& A, float2* d_lo, float2* m_lo, cudaStream_t s);
cudaError_t seq_update(const SeqArgs& A, cudaStream_t s);

// Every source one point component at its own position, and a beam shared by
// all tiles or none: its model is the same on every baseline.
bool peel_point_sources(const HdcSkyModel* h_sources, const RADec* h_positions, int num_sources, int beam_kind);
// Those models [source][timestep][channel] as FP32 (xx, yy, Re xy, Im xy) of
// the Hermitian B S B^H.
int peel_point_table(const HdcSkyModel* h_sources, int num_sources, const double* h_freqs, int num_freqs,
                     const double* h_lmsts, int num_timesteps, double latitude, int beam_kind, float4* d_table,
                     cudaStream_t s);

}  // namespace hdc

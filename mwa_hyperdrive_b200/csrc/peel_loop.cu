// Native peel loop: peel_gpu of mwa_hyperdrive (params/peel/gpu.rs:25-757)
// over libhdc's kernels, on one stream.
//
// Per pass and per source (Gauss-Seidel over sources, as the reference):
//   uvws_to   = xyzs_to_uvws(source position)
//   model     = the source predicted at its own phase centre with uvws_to (a
//               single point at its own position under a shared beam: one
//               Jones per timestep and channel, formed once for all passes)
//   traces of the residual rotated to the source (uvws_from -> uvws_to) with
//     model * iono(old consts) added, and of that model, averaged to low
//     resolution (time and channel groups) in one pass (seq_accumulate)
//   iono_loop from (0, 0, 1) on the low-resolution traces at the source's
//     low-resolution UVWs -> (da, db, dg)
//   consts    = (a + da, b + db, g * dg), reverted if |a| or |b| > 1e-3 or
//               g < 0 or g > 1.5 (gpu.rs:541-627)
//   residual  = rotated residual + model * iono(old) - model * iono(consts)
//               in one pass (seq_update)
//   uvws_from <- uvws_to
// then rotate back to the phase centre.  The constants stay on the device;
// the host reads them once at the end.

#include <cmath>
#include <memory>
#include <vector>

#include "peel.cuh"

using namespace hdc;

#define PEEL_CK(call)                                                        \
    do {                                                                     \
        cudaError_t e_ = (call);                                             \
        if (e_ != cudaSuccess) {                                             \
            set_error("hdc_peel_timeblock: %s: %s", #call, cudaGetErrorString(e_)); \
            return HDC_ERR_CUDA;                                             \
        }                                                                    \
    } while (0)

extern "C" int hdc_peel_timeblock(JonesF32* d_resid_tfb, const float* d_weights_tfb, int num_timesteps, int num_freqs,
                                  const double* h_freqs, const XYZ* h_tile_xyzs, int num_tiles, const double* h_lmsts,
                                  double average_lmst, RADec phase_centre, int num_sources,
                                  const HdcSkyModel* h_sources, const RADec* h_source_positions,
                                  IonoConsts* h_iono_consts, const HdcPeelParams* params, hdcStream_t stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (!d_resid_tfb || !d_weights_tfb || !h_freqs || !h_tile_xyzs || !h_lmsts || !params || num_tiles < 2 ||
        num_timesteps < 1 || num_freqs < 1 || num_sources < 0 || (num_sources > 0 && (!h_sources || !h_iono_consts ||
                                                                                      !h_source_positions))) {
        set_error("hdc_peel_timeblock: invalid arguments");
        return HDC_ERR_ARG;
    }
    const int favg = params->freq_average_factor;
    if (favg < 1 || num_freqs % favg != 0) {
        set_error("hdc_peel_timeblock: %d channels are not a multiple of the averaging factor %d", num_freqs, favg);
        return HDC_ERR_ARG;
    }
    if (num_sources == 0) return HDC_OK;
    const int nt = num_timesteps, nf = num_freqs, nbl = num_tiles * (num_tiles - 1) / 2, nlo = nf / favg;
    const size_t nvis = (size_t)nt * nf * nbl;

    // host-side tables
    std::vector<double> lam(nf), lam_lo(nlo);
    for (int f = 0; f < nf; f++) lam[f] = VEL_C / h_freqs[f];
    for (int k = 0; k < nlo; k++) {
        double sum = 0.0;
        for (int f = k * favg; f < (k + 1) * favg; f++) sum += h_freqs[f];
        lam_lo[k] = VEL_C / (sum / favg);
    }
    std::vector<XYZ> xyz_t((size_t)nt * num_tiles);
    for (int t = 0; t < nt; t++)
        for (int i = 0; i < num_tiles; i++) xyz_t[(size_t)t * num_tiles + i] = h_tile_xyzs[i];
    const int ns = num_sources;
    const bool points = peel_point_sources(h_sources, h_source_positions, ns, params->beam_kind);

    DevBuf b_lam, b_lam_lo, b_lmst, b_avg_lmst, b_xyz_t, b_from, b_to, b_uv_lo, b_model, b_point, b_dlo, b_mlo, b_w_lo,
        b_part, b_st, b_consts;
    PEEL_CK(b_lam.alloc(sizeof(double) * nf, s));
    PEEL_CK(b_lam_lo.alloc(sizeof(double) * nlo, s));
    PEEL_CK(b_lmst.alloc(sizeof(double) * nt, s));
    PEEL_CK(b_avg_lmst.alloc(sizeof(double), s));
    PEEL_CK(b_xyz_t.alloc(sizeof(XYZ) * xyz_t.size(), s));
    PEEL_CK(b_from.alloc(sizeof(UVW) * (size_t)nt * nbl, s));
    PEEL_CK(b_to.alloc(sizeof(UVW) * (size_t)nt * nbl, s));
    PEEL_CK(b_uv_lo.alloc(sizeof(UVW) * (size_t)ns * nbl, s));
    PEEL_CK(b_dlo.alloc(sizeof(float2) * (size_t)nlo * nbl, s));
    PEEL_CK(b_mlo.alloc(sizeof(float2) * (size_t)nlo * nbl, s));
    PEEL_CK(b_w_lo.alloc(sizeof(float) * (size_t)nlo * nbl, s));
    PEEL_CK(b_part.alloc(iono_partials_bytes(1, nbl), s));
    PEEL_CK(b_st.alloc(sizeof(IonoDev), s));
    PEEL_CK(b_consts.alloc(sizeof(IonoConsts) * 2 * ns, s));  // a pass's old and new constants, then the other way round
    PEEL_CK(cudaMemcpyAsync(b_lam.p, lam.data(), sizeof(double) * nf, cudaMemcpyHostToDevice, s));
    PEEL_CK(cudaMemcpyAsync(b_lam_lo.p, lam_lo.data(), sizeof(double) * nlo, cudaMemcpyHostToDevice, s));
    PEEL_CK(cudaMemcpyAsync(b_lmst.p, h_lmsts, sizeof(double) * nt, cudaMemcpyHostToDevice, s));
    PEEL_CK(cudaMemcpyAsync(b_avg_lmst.p, &average_lmst, sizeof(double), cudaMemcpyHostToDevice, s));
    PEEL_CK(cudaMemcpyAsync(b_xyz_t.p, xyz_t.data(), sizeof(XYZ) * xyz_t.size(), cudaMemcpyHostToDevice, s));
    PEEL_CK(cudaMemcpyAsync(b_consts.p, h_iono_consts, sizeof(IonoConsts) * ns, cudaMemcpyHostToDevice, s));
    PEEL_CK(k_weights_average(d_weights_tfb, b_w_lo.as<float>(), nt, nbl, nf, favg, s));
    PEEL_CK(iono_states_init(b_st.as<IonoDev>(), 1, s));

    // the sources' models: a table for points, else one modeller per source,
    // phase centre at the source (update_with_a_source with the source's
    // weighted position, gpu.rs:442)
    std::vector<std::unique_ptr<Modeller>> models;
    if (points) {
        PEEL_CK(b_point.alloc(sizeof(float4) * (size_t)ns * nt * nf, s));
        const int rc = peel_point_table(h_sources, ns, h_freqs, nf, h_lmsts, nt, params->array_latitude_rad,
                                        params->beam_kind, b_point.as<float4>(), s);
        if (rc) return rc;
    } else {
        PEEL_CK(b_model.alloc_plain(sizeof(JonesF32) * nvis));
        for (int i = 0; i < ns; i++) {
            HdcModeller* hm = nullptr;
            int rc = peel_modeller_new(&h_sources[i], h_tile_xyzs, num_tiles, h_freqs, num_freqs, h_source_positions[i],
                                       params, &hm);
            if (rc) return rc;
            models.emplace_back(reinterpret_cast<Modeller*>(hm));
        }
    }

    UVW* from = b_from.as<UVW>();
    UVW* to = b_to.as<UVW>();
    const XYZ* dxyz = b_xyz_t.as<XYZ>();
    const double* dlam = b_lam.as<double>();
    for (int i = 0; i < ns; i++)
        PEEL_CK(k_xyzs_to_uvws(dxyz, b_avg_lmst.as<double>(), b_uv_lo.as<UVW>() + (size_t)i * nbl, h_source_positions[i],
                               num_tiles, nbl, 1, s));
    const IonoConsts* result = b_consts.as<IonoConsts>();
    for (int pass = 0; pass < params->num_passes; pass++) {
        const IonoConsts* old = b_consts.as<IonoConsts>() + (pass & 1) * ns;
        IonoConsts* neu = b_consts.as<IonoConsts>() + ((pass + 1) & 1) * ns;
        PEEL_CK(k_xyzs_to_uvws(dxyz, b_lmst.as<double>(), from, phase_centre, num_tiles, nbl, nt, s));
        for (int i = 0; i < ns; i++) {
            PEEL_CK(k_xyzs_to_uvws(dxyz, b_lmst.as<double>(), to, h_source_positions[i], num_tiles, nbl, nt, s));
            if (!points) {
                PEEL_CK(cudaMemsetAsync(b_model.p, 0, sizeof(JonesF32) * nvis, s));
                for (int t = 0; t < nt; t++) {
                    int rc = models[i]->model_uvws(h_lmsts[t], to + (size_t)t * nbl,
                                                   b_model.as<JonesF32>() + (size_t)t * nf * nbl, s);
                    if (rc) return rc;
                }
            }
            const SeqArgs A = {d_resid_tfb, d_weights_tfb, points ? nullptr : b_model.as<JonesF32>(),
                               points ? b_point.as<float4>() + (size_t)i * nt * nf : nullptr,
                               old + i, neu + i, from, to, dlam, nt, nf, nbl, favg};
            PEEL_CK(seq_accumulate(A, b_dlo.as<float2>(), b_mlo.as<float2>(), s));
            PEEL_CK(iono_fit(b_dlo.as<float2>(), b_w_lo.as<float>(), b_mlo.as<float2>(), b_part.as<double>(),
                             b_st.as<IonoDev>(), old + i, neu + i, 1, nbl, nlo, params->num_loops,
                             b_uv_lo.as<UVW>() + (size_t)i * nbl, b_lam_lo.as<double>(), params->convergence, s));
            PEEL_CK(seq_update(A, s));
            std::swap(from, to);
        }
        PEEL_CK(k_xyzs_to_uvws(dxyz, b_lmst.as<double>(), to, phase_centre, num_tiles, nbl, nt, s));
        PEEL_CK(k_rotate(d_resid_tfb, nt, nbl, nf, from, to, dlam, s));
        result = neu;
    }
    PEEL_CK(cudaMemcpyAsync(h_iono_consts, result, sizeof(IonoConsts) * ns, cudaMemcpyDeviceToHost, s));
    PEEL_CK(cudaStreamSynchronize(s));
    return HDC_OK;
}

// Generated by rust/gen_bindings.py from include/hdc.h; do not edit.
#![allow(non_camel_case_types, non_snake_case, dead_code, unused_imports)]

use std::os::raw::{c_char, c_int, c_longlong, c_uchar, c_uint, c_ulonglong, c_void};

pub const HDC_NOALLOC_SCRATCH_BYTES: c_uint = 16777216;
pub const HDC_OK: c_int = 0;
pub const HDC_ERR_ARG: c_int = 1;
pub const HDC_ERR_CUDA: c_int = 2;
pub const HDC_ERR_ALLOC: c_int = 3;
pub const HDC_ERR_TIMEOUT: c_int = 4;
pub const HDC_ERR_UNSUPPORTED: c_int = 5;
pub const HDC_POINT: c_int = 0;
pub const HDC_GAUSSIAN: c_int = 1;
pub const HDC_SHAPELET: c_int = 2;
pub const HDC_FLUX_LIST: c_int = 0;
pub const HDC_FLUX_POWER_LAW: c_int = 1;
pub const HDC_FLUX_CURVED_POWER_LAW: c_int = 2;
pub const HDC_BEAM_NONE: c_int = 0;
pub const HDC_BEAM_ANALYTIC_DIPOLE: c_int = 1;
pub const HDC_BEAM_ANALYTIC_PER_TILE: c_int = 2;
pub const HDC_BEAM_FEE: c_int = 3;
pub const HDC_PREDICT_DIRECT: c_int = 0;
pub const HDC_PREDICT_TENSOR: c_int = 1;
pub const HDC_CAL_PLAIN: c_int = 0;
pub const HDC_CAL_COLLAPSED: c_int = 1;
pub const HDC_CAL_COLLAPSED_F32: c_int = 2;

#[repr(C)]
pub struct CUstream_st {
    _private: [u8; 0],
}

#[repr(C)]
pub struct HdcFeeBeam {
    _private: [u8; 0],
}

#[repr(C)]
pub struct HdcMlp {
    _private: [u8; 0],
}

#[repr(C)]
pub struct HdcModeller {
    _private: [u8; 0],
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct RADec {
    pub ra: f64,
    pub dec: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct HADec {
    pub ha: f64,
    pub dec: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct XYZ {
    pub x: f64,
    pub y: f64,
    pub z: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct UVW {
    pub u: f64,
    pub v: f64,
    pub w: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct LmnRime {
    pub l: f64,
    pub m: f64,
    pub n: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct GaussianParams {
    pub maj: f64,
    pub min: f64,
    pub pa: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct ShapeletCoeff {
    pub value: f64,
    pub n1: c_uchar,
    pub n2: c_uchar,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct ShapeletUV {
    pub u: f64,
    pub v: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct JonesF32 {
    pub j00_re: f32,
    pub j00_im: f32,
    pub j01_re: f32,
    pub j01_im: f32,
    pub j10_re: f32,
    pub j10_im: f32,
    pub j11_re: f32,
    pub j11_im: f32,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct JonesF64 {
    pub j00_re: f64,
    pub j00_im: f64,
    pub j01_re: f64,
    pub j01_im: f64,
    pub j10_re: f64,
    pub j10_im: f64,
    pub j11_re: f64,
    pub j11_im: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct Addresses {
    pub num_freqs: c_int,
    pub num_vis: c_int,
    pub num_baselines: c_int,
    pub d_freqs: *const f64,
    pub d_shapelet_basis_values: *const f64,
    pub num_unique_beam_freqs: c_int,
    pub d_tile_map: *const c_int,
    pub d_freq_map: *const c_int,
    pub d_tile_index_to_unflagged_tile_index_map: *const c_int,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct Points {
    pub num_power_laws: c_int,
    pub power_law_lmns: *const LmnRime,
    pub power_law_fds: *const JonesF64,
    pub power_law_sis: *const f64,
    pub num_curved_power_laws: c_int,
    pub curved_power_law_lmns: *const LmnRime,
    pub curved_power_law_fds: *const JonesF64,
    pub curved_power_law_sis: *const f64,
    pub curved_power_law_qs: *const f64,
    pub num_lists: c_int,
    pub list_lmns: *const LmnRime,
    pub list_fds: *const JonesF64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct Gaussians {
    pub num_power_laws: c_int,
    pub power_law_lmns: *const LmnRime,
    pub power_law_fds: *const JonesF64,
    pub power_law_sis: *const f64,
    pub power_law_gps: *const GaussianParams,
    pub num_curved_power_laws: c_int,
    pub curved_power_law_lmns: *const LmnRime,
    pub curved_power_law_fds: *const JonesF64,
    pub curved_power_law_sis: *const f64,
    pub curved_power_law_qs: *const f64,
    pub curved_power_law_gps: *const GaussianParams,
    pub num_lists: c_int,
    pub list_lmns: *const LmnRime,
    pub list_fds: *const JonesF64,
    pub list_gps: *const GaussianParams,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct Shapelets {
    pub num_power_laws: c_int,
    pub power_law_lmns: *const LmnRime,
    pub power_law_fds: *const JonesF64,
    pub power_law_sis: *const f64,
    pub power_law_gps: *const GaussianParams,
    pub power_law_shapelet_uvs: *const ShapeletUV,
    pub power_law_shapelet_coeffs: *const ShapeletCoeff,
    pub power_law_num_shapelet_coeffs: *const c_int,
    pub num_curved_power_laws: c_int,
    pub curved_power_law_lmns: *const LmnRime,
    pub curved_power_law_fds: *const JonesF64,
    pub curved_power_law_sis: *const f64,
    pub curved_power_law_qs: *const f64,
    pub curved_power_law_gps: *const GaussianParams,
    pub curved_power_law_shapelet_uvs: *const ShapeletUV,
    pub curved_power_law_shapelet_coeffs: *const ShapeletCoeff,
    pub curved_power_law_num_shapelet_coeffs: *const c_int,
    pub num_lists: c_int,
    pub list_lmns: *const LmnRime,
    pub list_fds: *const JonesF64,
    pub list_gps: *const GaussianParams,
    pub list_shapelet_uvs: *const ShapeletUV,
    pub list_shapelet_coeffs: *const ShapeletCoeff,
    pub list_num_shapelet_coeffs: *const c_int,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct IonoConsts {
    pub alpha: f64,
    pub beta: f64,
    pub gain: f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct HdcSkyModel {
    pub num_components: c_int,
    pub comp_type: *const c_int,
    pub ra: *const f64,
    pub dec: *const f64,
    pub maj: *const f64,
    pub min: *const f64,
    pub pa: *const f64,
    pub flux_type: *const c_int,
    pub si: *const f64,
    pub q: *const f64,
    pub fd_start: *const c_int,
    pub fd_count: *const c_int,
    pub fds: *const f64,
    pub coeff_start: *const c_int,
    pub coeff_count: *const c_int,
    pub coeff_n1: *const c_int,
    pub coeff_n2: *const c_int,
    pub coeff_value: *const f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct HdcFeeCoeffs {
    pub num_freqs: c_int,
    pub freqs_hz: *const u32,
    pub num_modes: c_int,
    pub modes: *const i32,
    pub num_freq_modes: *const i32,
    pub q: *const f64,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct HdcCalResult {
    pub num_iterations: c_int,
    pub converged: c_int,
    pub max_precision: f64,
    pub num_failed: c_int,
}

#[repr(C)]
#[derive(Debug, Clone, Copy)]
pub struct HdcPeelParams {
    pub num_passes: c_int,
    pub num_loops: c_int,
    pub convergence: f64,
    pub freq_average_factor: c_int,
    pub beam_kind: c_int,
    pub array_latitude_rad: f64,
    pub batch_size: c_int,
    pub fee_beam: *const HdcFeeBeam,
}

extern "C" {
    pub fn model_points(comps: *const Points, a: *const Addresses, d_uvws: *const UVW, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF32) -> *const c_char;
    pub fn model_points_noalloc(comps: *const Points, a: *const Addresses, d_uvws: *const UVW, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF32) -> *const c_char;
    pub fn model_points_f64out(comps: *const Points, a: *const Addresses, d_uvws: *const UVW, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF64) -> *const c_char;
    pub fn model_points_tc(comps: *const Points, a: *const Addresses, d_tile_xyzs: *const XYZ, lst_rad: f64, phase_centre: RADec, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF32) -> *const c_char;
    pub fn model_gaussians(comps: *const Gaussians, a: *const Addresses, d_uvws: *const UVW, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF32) -> *const c_char;
    pub fn model_gaussians_f64out(comps: *const Gaussians, a: *const Addresses, d_uvws: *const UVW, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF64) -> *const c_char;
    pub fn model_shapelets(comps: *const Shapelets, a: *const Addresses, d_uvws: *const UVW, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF32) -> *const c_char;
    pub fn model_shapelets_f64out(comps: *const Shapelets, a: *const Addresses, d_uvws: *const UVW, d_beam_jones: *const JonesF64, d_vis_fb: *mut JonesF64) -> *const c_char;
    pub fn model_autos(num_tiles: c_int, num_freqs: c_int, freqs: *const f64, points: *const Points, gaussians: *const Gaussians, shapelets: *const Shapelets, beam_jones: *const JonesF64, tile_map: *const c_int, freq_map: *const c_int, num_fee_freqs: c_int, tile_index_to_unflagged_tile_index_map: *const c_int, vis_fb: *mut JonesF32) -> *const c_char;
    pub fn xyzs_to_uvws(d_xyzs: *const XYZ, d_lmsts: *const f64, d_uvws: *mut UVW, pointing_centre: RADec, num_tiles: c_int, num_baselines: c_int, num_timesteps: c_int) -> *const c_char;
    pub fn rotate(vis_fb: *mut JonesF32, num_timesteps: c_int, num_baselines: c_int, num_freqs: c_int, uvws_from: *const UVW, uvws_to: *const UVW, lambdas: *const f64) -> *const c_char;
    pub fn average(d_high_res_vis: *const JonesF32, d_high_res_weights: *const f32, d_low_res_vis: *mut JonesF32, num_timesteps: c_int, num_baselines: c_int, num_freqs: c_int, freq_average_factor: c_int) -> *const c_char;
    pub fn iono_loop(d_vis_residual: *const JonesF32, d_vis_weights: *const f32, d_vis_model: *const JonesF32, d_vis_model_rotated: *mut JonesF32, d_iono_fits: *mut JonesF64, iono_consts: *mut IonoConsts, num_baselines: c_int, num_freqs: c_int, num_iterations: c_int, d_uvws: *const UVW, d_lambdas_m: *const f64, convergence: f64) -> *const c_char;
    pub fn subtract_iono(d_vis_residual: *mut JonesF32, d_vis_model: *const JonesF32, iono_consts: IonoConsts, old_iono_consts: IonoConsts, d_uvws: *const UVW, d_lambdas_m: *const f64, num_timesteps: c_int, num_baselines: c_int, num_freqs: c_int) -> *const c_char;
    pub fn add_model(d_vis_residual: *mut JonesF32, d_vis_model: *const JonesF32, iono_consts: IonoConsts, d_lambdas_m: *const f64, d_uvws: *const UVW, num_timesteps: c_int, num_freqs: c_int, num_baselines: c_int) -> *const c_char;
    pub fn get_gpu_device_info(device: c_int, name: *mut c_char, device_major: *mut c_int, device_minor: *mut c_int, total_global_mem: *mut usize, driver_version: *mut c_int, runtime_version: *mut c_int) -> *const c_char;
    pub fn hdc_last_error() -> *const c_char;
    pub fn hdc_device_info(buf: *mut c_char, buf_len: c_int) -> c_int;
    pub fn hdc_source_brightness(sky: *const HdcSkyModel, h_comp_source: *const c_int, num_sources: c_int, h_freqs: *const f64, num_freqs: c_int, lst_rad: f64, latitude_rad: f64, phase_centre: RADec, beam_kind: c_int, source_dist_cutoff_rad: f64, min_elevation_rad: f64, h_brightness: *mut f64) -> c_int;
    pub fn hdc_modeller_new(sky: *const HdcSkyModel, pols: c_int, h_unflagged_tile_xyzs: *const XYZ, num_tiles: c_int, h_freqs: *const f64, num_freqs: c_int, phase_centre: RADec, array_latitude_rad: f64, beam_kind: c_int, predict_form: c_int, out: *mut *mut HdcModeller) -> c_int;
    pub fn hdc_modeller_free(m: *mut HdcModeller);
    pub fn hdc_modeller_set_tile_xyzs(m: *mut HdcModeller, h_tile_xyzs: *const XYZ) -> c_int;
    pub fn hdc_modeller_set_tile_beams(m: *mut HdcModeller, h_dipole_gains: *const f64, freq_res_hz: f64) -> c_int;
    pub fn hdc_fee_beam_new(file: *const HdcFeeCoeffs, h_freqs_hz: *const u32, num_freqs: c_int, h_delays: *const u32, h_amps: *const f64, num_tiles: c_int, num_amps: c_int, norm_to_zenith: c_int, out: *mut *mut HdcFeeBeam) -> c_int;
    pub fn hdc_fee_beam_free(b: *mut HdcFeeBeam);
    pub fn hdc_fee_beam_num_unique_tiles(b: *const HdcFeeBeam) -> c_int;
    pub fn hdc_fee_beam_num_unique_freqs(b: *const HdcFeeBeam) -> c_int;
    pub fn hdc_fee_beam_tile_map(b: *const HdcFeeBeam) -> *const c_int;
    pub fn hdc_fee_beam_freq_map(b: *const HdcFeeBeam) -> *const c_int;
    pub fn hdc_fee_beam_host_maps(b: *const HdcFeeBeam, h_tile_map: *mut c_int, h_freq_map: *mut c_int) -> c_int;
    pub fn hdc_fee_calc_jones(b: *const HdcFeeBeam, d_az_rad: *const f64, d_za_rad: *const f64, num_directions: c_int, d_latitude_rad: *const f64, iau_order: c_int, d_jones: *mut JonesF64, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_modeller_set_fee_beam(m: *mut HdcModeller, b: *const HdcFeeBeam) -> c_int;
    pub fn hdc_source_brightness_fee(sky: *const HdcSkyModel, h_comp_source: *const c_int, num_sources: c_int, h_freqs: *const f64, num_freqs: c_int, lst_rad: f64, latitude_rad: f64, phase_centre: RADec, beam: *const HdcFeeBeam, source_dist_cutoff_rad: f64, min_elevation_rad: f64, h_brightness: *mut f64) -> c_int;
    pub fn hdc_modeller_model_timestep_with(m: *mut HdcModeller, lst_rad: f64, d_vis_fb: *mut JonesF32, h_uvws_out: *mut UVW, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_modeller_model_timestep_with_f64(m: *mut HdcModeller, lst_rad: f64, d_vis_fb: *mut JonesF64, h_uvws_out: *mut UVW, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_modeller_model_timestep_with_host(m: *mut HdcModeller, lst_rad: f64, h_vis_fb: *mut JonesF32, h_uvws_out: *mut UVW, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_modeller_update_with_a_source(m: *mut HdcModeller, source: *const HdcSkyModel, phase_centre: RADec) -> c_int;
    pub fn hdc_modeller_model_timestep_autos_with(m: *mut HdcModeller, lst_rad: f64, d_vis_fb: *mut JonesF32, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_kernel_launches() -> c_longlong;
    pub fn hdc_kernel_error_string(word: c_int) -> *const c_char;
    pub fn hdc_test_stall_next_predict(wait_ns: c_ulonglong) -> c_int;
    pub fn hdc_test_limit_scratch(bytes: c_ulonglong) -> c_int;
    pub fn hdc_modeller_set_profiling(m: *mut HdcModeller, enable: c_int) -> c_int;
    pub fn hdc_modeller_profile(m: *mut HdcModeller, out_ms: *mut f64, reset: c_int) -> c_int;
    pub fn hdc_probe_fp64_gflops(out_gflops: *mut f64) -> c_int;
    pub fn hdc_probe_fp32_gflops(out_gflops: *mut f64) -> c_int;
    pub fn hdc_calibrate_timeblock(d_data_tfb: *const JonesF32, d_model_tfb: *const JonesF32, num_timesteps: c_int, timeblock_start: c_int, timeblock_end: c_int, num_chanblocks: c_int, num_baselines: c_int, d_di_jones: *mut JonesF64, max_iterations: c_int, stop_threshold: f64, min_threshold: f64, pols: c_int, h_results: *mut HdcCalResult, form: c_int, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_calibrate_chanblocks(d_data_tfb: *const JonesF32, d_model_tfb: *const JonesF32, num_timesteps: c_int, timeblock_start: c_int, timeblock_end: c_int, num_chanblocks: c_int, num_baselines: c_int, d_di_jones: *mut JonesF64, max_iterations: c_int, stop_threshold: f64, min_threshold: f64, pols: c_int, h_chanblock_list: *const c_int, num_listed: c_int, h_results: *mut HdcCalResult, form: c_int, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_calibrate_timeblocks(d_data_tfb: *const JonesF32, d_model_tfb: *const JonesF32, num_timesteps: c_int, h_timeblock_bounds: *const c_int, num_timeblocks: c_int, num_chanblocks: c_int, num_baselines: c_int, d_di_jones: *mut JonesF64, max_iterations: c_int, stop_threshold: f64, min_threshold: f64, pols: c_int, h_results: *mut HdcCalResult, form: c_int, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_calibration_residuals(d_data_tfb: *const JonesF32, d_model_tfb: *const JonesF32, num_timesteps: c_int, timeblock_start: c_int, timeblock_end: c_int, num_chanblocks: c_int, num_baselines: c_int, d_di_jones: *const JonesF64, h_residuals: *mut f64, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_mlp_new(num_layers: c_int, dims: *const c_int, residual_offset: c_int, seed: c_ulonglong, out: *mut *mut HdcMlp) -> c_int;
    pub fn hdc_mlp_free(m: *mut HdcMlp);
    pub fn hdc_mlp_num_params(m: *mut HdcMlp) -> c_longlong;
    pub fn hdc_mlp_get_params(m: *mut HdcMlp, h_out: *mut f32) -> c_int;
    pub fn hdc_mlp_set_params(m: *mut HdcMlp, h_in: *const f32) -> c_int;
    pub fn hdc_mlp_forward(m: *mut HdcMlp, d_x: *const f32, batch: c_int, d_y: *mut f32, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_mlp_gradients(m: *mut HdcMlp, d_x: *const f32, d_target: *const f32, batch: c_int, h_grads: *mut f32, h_loss: *mut f64, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_mlp_train_step(m: *mut HdcMlp, d_x: *const f32, d_target: *const f32, batch: c_int, lr: f32, h_loss: *mut f64, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_warmstart_features(d_prev_tc: *const JonesF64, num_tiles: c_int, num_chanblocks: c_int, d_x: *mut f32, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_warmstart_judge(d_data_tfb: *const JonesF32, d_model_tfb: *const JonesF32, num_timesteps: c_int, timeblock_start: c_int, timeblock_end: c_int, num_chanblocks: c_int, num_tiles: c_int, d_proposal_tc: *const JonesF64, d_start_tc: *mut JonesF64, d_use: *mut c_int, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_warmstart_propose(mlp: *mut HdcMlp, d_prev_tc: *const JonesF64, num_tiles: c_int, num_chanblocks: c_int, d_data_tfb: *const JonesF32, d_model_tfb: *const JonesF32, num_timesteps: c_int, timeblock_start: c_int, timeblock_end: c_int, d_start_tc: *mut JonesF64, d_use: *mut c_int, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_peel_timeblock(d_resid_tfb: *mut JonesF32, d_weights_tfb: *const f32, num_timesteps: c_int, num_freqs: c_int, h_freqs: *const f64, h_tile_xyzs: *const XYZ, num_tiles: c_int, h_lmsts: *const f64, average_lmst: f64, phase_centre: RADec, num_sources: c_int, h_sources: *const HdcSkyModel, h_source_positions: *const RADec, h_iono_consts: *mut IonoConsts, params: *const HdcPeelParams, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_peel_timeblock_batched(d_resid_tfb: *mut JonesF32, d_weights_tfb: *const f32, num_timesteps: c_int, num_freqs: c_int, h_freqs: *const f64, h_tile_xyzs: *const XYZ, num_tiles: c_int, h_lmsts: *const f64, average_lmst: f64, phase_centre: RADec, num_sources: c_int, h_sources: *const HdcSkyModel, h_source_positions: *const RADec, h_iono_consts: *mut IonoConsts, params: *const HdcPeelParams, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_peel_batched_tuning(block_bins: *mut c_int, block_sources: *mut c_int, ms: *mut f32) -> c_int;
    pub fn hdc_scale_by_weights(d_data_tfb: *mut JonesF32, d_model_tfb: *mut JonesF32, d_weights_tfb: *const f32, num_timesteps: c_int, num_chanblocks: c_int, num_baselines: c_int, d_baseline_weights: *const f64, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_vis_average(d_from_tfb: *const JonesF32, d_weights_from_tfb: *const f32, num_timesteps: c_int, num_freqs: c_int, num_baselines: c_int, h_flagged_chanblocks: *const c_int, num_flagged: c_int, d_to_fb: *mut JonesF32, d_weights_to_fb: *mut f32, num_chanblocks: c_int, stream: *mut CUstream_st) -> c_int;
    pub fn hdc_into_cal_sols(d_di_jones: *const JonesF64, num_timeblocks: c_int, num_unflagged_tiles: c_int, num_unflagged_chanblocks: c_int, h_flagged_tiles: *const c_int, num_flagged_tiles: c_int, h_flagged_chanblocks: *const c_int, num_flagged_chanblocks: c_int, pols: c_int, d_out: *mut JonesF64, stream: *mut CUstream_st) -> c_int;
}

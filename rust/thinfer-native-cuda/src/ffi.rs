//! Raw bindings of libthinfer_nvfp4.so (include/thinfer_nvfp4.h). GENERATED by gen_ffi.py: edit the header and the
//! generator, not this file. A safe wrapper crate maps `PreparedWeight::Nvfp4` and the NVFP4 arm of
//! `Block::dispatch_matmul_site_diag` to `tnf_linear_nvfp4`, `WeightResidency` uploads to `tnf_stream_upload`,
//! and an awaited `Backend::submit` to `tnf_sync`.
#![allow(non_camel_case_types, dead_code)]
use std::os::raw::{c_char, c_void};

#[repr(C)] pub struct TnfCtx { _private: [u8; 0] }
#[repr(C)] pub struct TnfStack { _private: [u8; 0] }
#[repr(C)] pub struct TnfGguf { _private: [u8; 0] }

/// BufRef (thinfer-core/src/backend/mod.rs:12-33): non-owning {id, offset, len} view.
#[repr(C)] #[derive(Clone, Copy, Default)]
pub struct TnfBuf { pub id: u64, pub offset: u64, pub len: u64 }

#[repr(C)] #[derive(Clone, Copy, Default)]
pub struct TnfLinearArgs {
    pub m: u32, pub n: u32, pub k: u32,
    pub a_global: f32, pub w_global: f32,
    pub a_bf16: TnfBuf, pub w_codes: TnfBuf, pub w_scales: TnfBuf, pub bias_bf16: TnfBuf,
    pub gate_bf16: TnfBuf, pub residual_bf16: TnfBuf, pub out_bf16: TnfBuf,
    pub act: u32, pub parity_mode: u32, pub n_offset: u32, pub ldo: u32, pub flags: u32,
    pub out_global: f32,
    pub out_codes: TnfBuf, pub out_scales: TnfBuf, pub w_dense: TnfBuf,
}

#[repr(C)] #[derive(Clone, Copy, Default)]
pub struct TnfNormQuantArgs {
    pub m: u32, pub k: u32, pub eps: f32, pub mod_bias: f32,
    pub x_bf16: TnfBuf, pub scale_bf16: TnfBuf, pub shift_bf16: TnfBuf, pub out_bf16: TnfBuf,
    pub out_codes: TnfBuf, pub out_scales: TnfBuf,
    pub out_global: f32, pub parity_mode: u32,
}

#[repr(C)] #[derive(Clone, Copy, Default)]
pub struct TnfSdpaArgs {
    pub b: u32, pub s_q: u32, pub s_k: u32, pub h_q: u32, pub h_kv: u32, pub d: u32,
    pub scale: f32, pub mask_mode: u32,
    pub q: TnfBuf, pub k: TnfBuf, pub v: TnfBuf, pub out: TnfBuf,
    pub flags: u32, pub out_global: f32, pub out_codes: TnfBuf, pub out_scales: TnfBuf,
    pub q_ld: u32, pub kv_ld: u32,
}

#[repr(C)] #[derive(Clone, Copy, Default)]
pub struct TnfStackLinear { pub n: u32, pub k: u32, pub act: u32, pub has_bias: u32, pub input: u32, pub stream_id: u32 }

/// DenseActSites (thinfer-models/src/common/block.rs:470-479).
#[repr(C)] #[derive(Clone, Copy, Default)]
pub struct TnfDenseActSites { pub qkv: u32, pub qkv_self: u32, pub proj: u32, pub ffn_up: u32, pub ffn_down: u32 }

#[repr(C)]
pub struct TnfGgufTensorInfo {
    pub name: *const c_char, pub n_dims: u32, pub dims: [u64; 8], pub ggml_type: u32,
    pub offset: u64, pub size: u64, pub on_disk_bytes: u64,
}

/// WeightReader (thinfer-core/src/weight.rs:57-77) as function pointers over an opaque `user`.
#[repr(C)] #[derive(Clone, Copy)]
pub struct TnfReader {
    pub user: *mut c_void,
    pub len: Option<unsafe extern "C" fn(user: *mut c_void) -> u64>,
    pub read_at: Option<unsafe extern "C" fn(user: *mut c_void, offset: u64, dst: *mut c_void, n: u64) -> i32>,
    pub will_read: Option<unsafe extern "C" fn(user: *mut c_void, offset: u64, n: u64)>,
    pub close: Option<unsafe extern "C" fn(user: *mut c_void)>,
}

pub const TNF_READER_DEFAULT_HINTS: u32 = 0xFFFF_FFFF;
pub const TNF_OK: i32 = 0;
pub const TNF_ERR_UNKNOWN_BUFFER: i32 = -1;
pub const TNF_ERR_ALLOCATE_OOM: i32 = -2;
pub const TNF_ERR_BUDGET_EXCEEDED: i32 = -3;
pub const TNF_ERR_INVALID_ARGUMENT: i32 = -4;
pub const TNF_ERR_LAUNCH: i32 = -5;
pub const TNF_ERR_TIMEOUT: i32 = -6;
pub const TNF_ERR_NCCL: i32 = -7;
pub const TNF_LINEAR_A_PREQUANTIZED: u32 = 1;
pub const TNF_LINEAR_SCATTER_PEERS: u32 = 2;
pub const TNF_LINEAR_OUT_NVFP4: u32 = 4;
pub const TNF_LINEAR_NO_BF16_OUT: u32 = 8;
pub const TNF_LINEAR_MULTICAST_OUT: u32 = 16;
pub const TNF_LINEAR_DENSE_ACT: u32 = 32;
pub const TNF_LINEAR_SWIGLU: u32 = 64;
pub const TNF_SDPA_OUT_NVFP4: u32 = 1;
pub const TNF_SDPA_NO_BF16_OUT: u32 = 2;

#[link(name = "thinfer_nvfp4")]
extern "C" {
    pub fn tnf_create(device: i32, vram_budget_bytes: u64, out: *mut *mut TnfCtx) -> i32;
    pub fn tnf_destroy(ctx: *mut TnfCtx) -> i32;
    pub fn tnf_last_error() -> *const c_char;
    pub fn tnf_abi_version() -> u32;
    pub fn tnf_alloc(ctx: *mut TnfCtx, bytes: u64, category: i32, id: *mut u64) -> i32;
    pub fn tnf_free(ctx: *mut TnfCtx, id: u64) -> i32;
    pub fn tnf_write(ctx: *mut TnfCtx, id: u64, dst_off: u64, src: *const c_void, n: u64) -> i32;
    pub fn tnf_read(ctx: *mut TnfCtx, id: u64, off: u64, dst: *mut c_void, n: u64) -> i32;
    pub fn tnf_copy(ctx: *mut TnfCtx, src_id: u64, src_off: u64, dst_id: u64, dst_off: u64, n: u64) -> i32;
    pub fn tnf_buf_ptr(ctx: *mut TnfCtx, id: u64, device_ptr: *mut *mut c_void, bytes: *mut u64) -> i32;
    pub fn tnf_sync(ctx: *mut TnfCtx, timeout_ms: u32) -> i32;
    pub fn tnf_mem_snapshot(ctx: *mut TnfCtx, out: *mut u64) -> i32;
    pub fn tnf_reclaimed_bytes(ctx: *mut TnfCtx, bytes: *mut u64) -> i32;
    pub fn tnf_ws_alloc(ctx: *mut TnfCtx, bytes: u64, id: *mut u64) -> i32;
    pub fn tnf_ws_release(ctx: *mut TnfCtx, id: u64) -> i32;
    pub fn tnf_ws_drain(ctx: *mut TnfCtx, freed_bytes: *mut u64) -> i32;
    pub fn tnf_ws_stats(ctx: *mut TnfCtx, out: *mut u64) -> i32;
    pub fn tnf_set_transient_reserve(ctx: *mut TnfCtx, bytes: u64) -> i32;
    pub fn tnf_set_device_wait_limit(ctx: *mut TnfCtx, sm_cycles: u64) -> i32;
    pub fn tnf_selftest_stalled_wait(ctx: *mut TnfCtx) -> i32;
    pub fn tnf_streams(ctx: *mut TnfCtx, compute_stream: *mut *mut c_void, copy_stream: *mut *mut c_void) -> i32;
    pub fn tnf_quantize_weight(ctx: *mut TnfCtx, w_src: TnfBuf, src_dtype: i32, n: u32, k: u32, codes: TnfBuf, scales: TnfBuf, global_scale: *mut f32) -> i32;
    pub fn tnf_load_weight(ctx: *mut TnfCtx, w_host: *const c_void, src_dtype: i32, n: u32, k: u32, bias_host: *const u16, codes_id: *mut u64, scales_id: *mut u64, bias_id: *mut u64, global_scale: *mut f32) -> i32;
    pub fn tnf_device_scales_bytes(rows: u32, k: u32) -> u64;
    pub fn tnf_prepare_scales(ctx: *mut TnfCtx, scales_canonical: TnfBuf, rows: u32, k: u32, scales_device: TnfBuf) -> i32;
    pub fn tnf_quantize_act(ctx: *mut TnfCtx, a_bf16: TnfBuf, m: u32, k: u32, global_scale: f32, scales_layout: i32, codes: TnfBuf, scales: TnfBuf, global_scale_used: *mut f32) -> i32;
    pub fn tnf_site_linear_flags(policy: *const TnfDenseActSites, site: i32) -> u32;
    pub fn tnf_linear_nvfp4(ctx: *mut TnfCtx, args: *const TnfLinearArgs) -> i32;
    pub fn tnf_prepare_dense(ctx: *mut TnfCtx, w_codes: TnfBuf, w_scales_device: TnfBuf, n: u32, k: u32, out_bf16: TnfBuf) -> i32;
    pub fn tnf_norm_modulate_quantize(ctx: *mut TnfCtx, args: *const TnfNormQuantArgs) -> i32;
    pub fn tnf_linear_nvfp4_noalloc(ctx: *mut TnfCtx, args: *const TnfLinearArgs) -> i32;
    pub fn tnf_noalloc_scratch_bytes() -> u64;
    pub fn tnf_quantize_act_shared(ctx: *mut TnfCtx, a_bf16: TnfBuf, m: u32, k: u32, global_scale: f32) -> i32;
    pub fn tnf_gemm_nvfp4(ctx: *mut TnfCtx, args: *const TnfLinearArgs, a_codes: TnfBuf, a_scales_device: TnfBuf) -> i32;
    pub fn tnf_sdpa(ctx: *mut TnfCtx, args: *const TnfSdpaArgs) -> i32;
    pub fn tnf_host_register(ctx: *mut TnfCtx, host_ptr: *mut c_void, bytes: u64, host_id: *mut u64) -> i32;
    pub fn tnf_host_ptr(ctx: *mut TnfCtx, host_id: u64, ptr: *mut *mut c_void, bytes: *mut u64) -> i32;
    pub fn tnf_host_release(ctx: *mut TnfCtx, host_id: u64) -> i32;
    pub fn tnf_stream_upload(ctx: *mut TnfCtx, host_id: u64, host_off: u64, dst_id: u64, dst_off: u64, n: u64, event: *mut u64) -> i32;
    pub fn tnf_wait_event(ctx: *mut TnfCtx, event: u64) -> i32;
    pub fn tnf_stream_download(ctx: *mut TnfCtx, src_id: u64, src_off: u64, host_id: u64, host_off: u64, n: u64, event: *mut u64) -> i32;
    pub fn tnf_event_sync(ctx: *mut TnfCtx, event: u64) -> i32;
    pub fn tnf_copy_after_compute(ctx: *mut TnfCtx) -> i32;
    pub fn tnf_stack_record_bytes(n: u32, k: u32) -> u64;
    pub fn tnf_stack_record_offsets(n: u32, k: u32, out: *mut u64) -> i32;
    pub fn tnf_stack_create(ctx: *mut TnfCtx, layers: u32, n_linears: u32, linears: *const TnfStackLinear, n_streams: u32, m_rows: *const u32, hidden: u32, host_id: u64, weight_budget_bytes: u64, ring_slots: u32, out: *mut *mut TnfStack) -> i32;
    pub fn tnf_stack_step(st: *mut TnfStack, x_ids: *const u64, aux_ids: *const u64, out_ids: *const u64, a_global: f32) -> i32;
    pub fn tnf_stack_stats(st: *mut TnfStack, out: *mut u64) -> i32;
    pub fn tnf_stack_evict_all(st: *mut TnfStack) -> i32;
    pub fn tnf_stack_restore(st: *mut TnfStack, weight_budget_bytes: u64) -> i32;
    pub fn tnf_stack_destroy(st: *mut TnfStack) -> i32;
    pub fn tnf_mmap_open(path: *const c_char, out: *mut TnfReader) -> i32;
    pub fn tnf_mmap_stats(r: *const TnfReader, out: *mut u64) -> i32;
    pub fn tnf_reader_view(inner: *const TnfReader, base: u64, len: u64, out: *mut TnfReader) -> i32;
    pub fn tnf_reader_close(r: *mut TnfReader);
    pub fn tnf_reader_read(r: *const TnfReader, offset: u64, n: u64, dst: *mut c_void, chunk_bytes: u64, hint_chunks: u32) -> i32;
    pub fn tnf_reader_read_to_arena(ctx: *mut TnfCtx, r: *const TnfReader, offset: u64, n: u64, host_id: u64, host_off: u64, chunk_bytes: u64, hint_chunks: u32) -> i32;
    pub fn tnf_upload_from_reader(ctx: *mut TnfCtx, r: *const TnfReader, src_offset: u64, total: u64, dst: TnfBuf, chunk_bytes: u64, hint_chunks: u32, event: *mut u64) -> i32;
    pub fn tnf_gguf_parse(buf: *const c_void, len: u64, out: *mut *mut TnfGguf, need_at: *mut u64) -> i32;
    pub fn tnf_gguf_free(h: *mut TnfGguf) -> i32;
    pub fn tnf_gguf_info(h: *const TnfGguf, out: *mut u64) -> i32;
    pub fn tnf_gguf_tensor(h: *const TnfGguf, index: u64, file_size: u64, out: *mut TnfGgufTensorInfo) -> i32;
    pub fn tnf_ggml_type_label(ggml_type: u32) -> *const c_char;
    pub fn tnf_comm_unique_id(unique_id_128: *mut c_void) -> i32;
    pub fn tnf_comm_init(ctx: *mut TnfCtx, world: i32, rank: i32, unique_id_128: *const c_void) -> i32;
    pub fn tnf_all_gather_cols(ctx: *mut TnfCtx, out_bf16: TnfBuf, m: u32, n_total: u32, n_local: u32) -> i32;
    pub fn tnf_all_gather_nvfp4(ctx: *mut TnfCtx, codes: TnfBuf, scales: TnfBuf, m: u32, n_total: u32, n_local: u32) -> i32;
    pub fn tnf_ipc_export(ctx: *mut TnfCtx, id: u64, handle_64: *mut c_void) -> i32;
    pub fn tnf_peer_outputs(ctx: *mut TnfCtx, set: i32, n_peers: i32, handles_64xn: *const c_void) -> i32;
    pub fn tnf_scatter_rows(ctx: *mut TnfCtx, set: i32, out_bf16: TnfBuf, row0: u32, rows: u32, n_offset: u32, n: u32, ldo: u32) -> i32;
    pub fn tnf_push_peers(ctx: *mut TnfCtx, set: i32, src: TnfBuf, dst_offset: u64, self_dst: TnfBuf) -> i32;
    pub fn tnf_compute_after_push(ctx: *mut TnfCtx) -> i32;
    pub fn tnf_interleave_cols(ctx: *mut TnfCtx, gathered: TnfBuf, rank_stride: u64, src_row_bytes: u32, world: u32, out: TnfBuf, out_row_bytes: u32, rows: u32, local_row_bytes: u32) -> i32;
    pub fn tnf_compute_after_copy(ctx: *mut TnfCtx) -> i32;
    pub fn tnf_comm_barrier(ctx: *mut TnfCtx) -> i32;
    pub fn tnf_import_symmetric(ctx: *mut TnfCtx, local_ptr: *mut c_void, multicast_ptr: *mut c_void, bytes: u64, category: i32, id: *mut u64) -> i32;
    pub fn tnf_multicast_copy(ctx: *mut TnfCtx, src: TnfBuf, dst_id: u64, dst_off: u64, n: u64) -> i32;
}

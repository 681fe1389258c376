"""Writes src/ffi.rs: the `extern "C"` declarations of every function in include/thinfer_nvfp4.h.

    python rust/thinfer-native-cuda/gen_ffi.py

The struct definitions (`#[repr(C)]`) are written by hand in the template below and must follow the
header; the function list is taken from the header's prototypes, so the two cannot drift apart
(tests/test_abi.py compares the generated file with the header's symbol list)."""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
HEADER = os.path.join(HERE, "..", "..", "include", "thinfer_nvfp4.h")

TYPES = {
    "int32_t": "i32", "uint32_t": "u32", "uint64_t": "u64", "int": "i32", "float": "f32", "uint16_t": "u16", "void": "c_void",
    "tnf_ctx": "TnfCtx", "tnf_buf": "TnfBuf", "tnf_linear_args": "TnfLinearArgs", "tnf_norm_quant_args": "TnfNormQuantArgs",
    "tnf_stack": "TnfStack", "tnf_stack_linear": "TnfStackLinear", "tnf_gguf": "TnfGguf",
    "tnf_gguf_tensor_info": "TnfGgufTensorInfo", "tnf_dense_act_sites": "TnfDenseActSites", "char": "c_char",
    "tnf_reader": "TnfReader", "tnf_sdpa_args": "TnfSdpaArgs",
}

HEAD = '''//! Raw bindings of libthinfer_nvfp4.so (include/thinfer_nvfp4.h). GENERATED by gen_ffi.py: edit the header and the
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
'''


def rust_type(c: str) -> str:
    c = c.strip()
    const = c.startswith("const ")
    c = c.replace("const ", "").strip()
    stars = c.count("*")
    base = c.replace("*", "").strip()
    t = TYPES[base]
    for _ in range(stars):
        t = ("*const " if const else "*mut ") + t
    return t


def prototypes(text: str):
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    for m in re.finditer(r"^([a-z_0-9 ]+?[\s\*]+)(tnf_[a-z0-9_]+)\s*\(([^;{]*?)\)\s*;", text, flags=re.M | re.S):
        ret, name, args = m.group(1).strip(), m.group(2), " ".join(m.group(3).split())
        yield ret, name, args


def main():
    out = [HEAD]
    for ret, name, args in prototypes(open(HEADER).read()):
        params = []
        if args and args != "void":
            for a in args.split(","):
                a = a.strip()
                arr = re.match(r"(.*?)(\w+)\[(\d*)\]$", a)
                if arr:  # C array parameter = pointer
                    ctype, pname = arr.group(1).strip() + "*", arr.group(2)
                else:
                    mm = re.match(r"(.*?)(\w+)$", a)
                    ctype, pname = mm.group(1).strip(), mm.group(2)
                if pname in ("type", "in", "ref", "move"):
                    pname += "_"
                params.append(f"{pname}: {rust_type(ctype)}")
        r = "" if ret == "void" else f" -> {rust_type(ret)}"
        out.append(f"    pub fn {name}({', '.join(params)}){r};\n")
    out.append("}\n")
    dst = os.path.join(HERE, "src", "ffi.rs")
    open(dst, "w").write("".join(out))
    print(dst)


if __name__ == "__main__":
    main()

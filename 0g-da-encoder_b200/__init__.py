"""B200 blob encoder for the 0G DA encoder path — Python host binding.

Mirrors the reference's host interface over the C ABI of
include/zg_encoder.h (ctypes):

  reference (0glabs/0g-da-encoder)                   here
  -------------------------------------------------  ---------------------------
  constants BLOB_ROW_LOG/BLOB_COL_LOG/...             Dims
  (crates/encoder/src/constants.rs:14-28)
  RawData::try_from(&[u8]) (raw_data.rs:55-72)        RawData.try_from(bytes)
  EncoderError::TooLargeBlob (encoder/error.rs:3-6)   TooLargeBlob
  ZgEncoderParams::from_dir_mont (blob/encode.rs:114) ZgEncoderParams.from_dir_mont
  PowerTau::setup_inner(Some(tau)) + from_pp          ZgEncoderParams.from_seed
  EncodedBlob::build/get_row/get_commitment/...       EncodedBlob
  (crates/encoder/src/encoder/blob.rs:32-62)
  EncoderService::process_data (grpc/src/service.rs)  EncoderService.process_data
  EncodeBlobReply (grpc/proto/encoder.proto:16-22)    EncodeBlobReply

All compute runs in the CUDA library; there is no CPU fallback. Importing
works without a GPU; creating params requires one.
"""
import ctypes
import os
from dataclasses import dataclass, field
from typing import List

from . import build as _build

__all__ = [
    "Dims", "RawData", "EncoderError", "TooLargeBlob", "ZgEncoderParams", "EncodedBlob",
    "EncodeBlobReply", "EncoderService", "lib", "LIB_PATH", "C_ABI_FUNCTIONS", "recover_from_da_slice",
    "RecoveryError", "Ticket", "LightEncodedSlice",
]

LIB_PATH = _build.LIB
_lib = None

ZG_OK = 0
ZG_ERR_TOO_LARGE_BLOB = 1
ZG_ERR_RECOVERY = 2
ZG_ERR_TIMEOUT = 3
ZG_REQ_ENCODE = 0
ZG_REQ_RECOVER = 1


class _Config(ctypes.Structure):
    _fields_ = [
        ("log_row", ctypes.c_uint32),
        ("log_col", ctypes.c_uint32),
        ("tau_seed", ctypes.c_uint64),
        ("params_dir", ctypes.c_char_p),
        ("device", ctypes.c_int),
        ("msm_window_bits", ctypes.c_uint32),
    ]


class _DeviceBlob(ctypes.Structure):
    _fields_ = [
        ("encoded_data", ctypes.c_void_p),
        ("slices", ctypes.c_void_p),
        ("slice_size", ctypes.c_size_t),
        ("amt_outputs", ctypes.c_void_p),
        ("roots", ctypes.c_void_p),
        ("file_root", ctypes.c_void_p),
    ]


# ZG_MSM_PRODUCT_IMAD / _HYBRID / _FP64 / _W28 / _W28_HYBRID
MSM_PRODUCTS = ("imad", "hybrid", "fp64", "w28", "w28_hybrid")
MSM_TASK_SIZES = (32, 48, 64, 96)
MSM_WIDE_MAX = 6


class _Tuning(ctypes.Structure):
    """zg_tuning (include/zg_encoder.h)."""
    _fields_ = [("msm_product", ctypes.c_uint32), ("msm_task", ctypes.c_uint32),
                ("msm_wide_classes", ctypes.c_uint32), ("ntt_cols_per_cta", ctypes.c_uint32),
                ("ntt_threads", ctypes.c_uint32), ("msm_ms", ctypes.c_float * len(MSM_PRODUCTS)),
                ("task_ms", ctypes.c_float * len(MSM_TASK_SIZES)), ("wide_ms", ctypes.c_float * (MSM_WIDE_MAX + 1)),
                ("ntt_ms", ctypes.c_float * 9), ("msm_wide_lines", ctypes.c_uint32),
                ("msm_wide_avail", ctypes.c_uint32)]


def _tuning_dict(t):
    return {"msm_product": MSM_PRODUCTS[t.msm_product], "msm_task": t.msm_task,
            "msm_wide_classes": t.msm_wide_classes, "ntt_cols_per_cta": t.ntt_cols_per_cta,
            "ntt_threads": t.ntt_threads, "msm_ms": [round(x, 4) for x in t.msm_ms],
            "task_ms": [round(x, 4) for x in t.task_ms], "wide_ms": [round(x, 4) for x in t.wide_ms],
            "ntt_ms": [round(x, 4) for x in t.ntt_ms], "msm_wide_lines": t.msm_wide_lines,
            "msm_wide_avail": t.msm_wide_avail}


MAX_FUSED_BLOBS = 2  # ZG_MAX_FUSED_BLOBS


class _PipelineConfig(ctypes.Structure):
    """zg_pipeline_config (include/zg_encoder.h)."""
    _fields_ = [("max_units", ctypes.c_uint32), ("blobs_per_launch", ctypes.c_uint32),
                ("reserve_mib", ctypes.c_uint32)]


class _PipelineStats(ctypes.Structure):
    """zg_pipeline_stats (include/zg_encoder.h)."""
    _fields_ = [("units", ctypes.c_uint64), ("launches", ctypes.c_uint64 * MAX_FUSED_BLOBS),
                ("max_in_flight", ctypes.c_uint64), ("recoveries", ctypes.c_uint64),
                ("unit_bytes", ctypes.c_uint64)]


_P = ctypes.c_void_p
_SZ = ctypes.c_size_t


class _Request(ctypes.Structure):
    """zg_request (include/zg_encoder.h)."""
    _fields_ = [("kind", ctypes.c_int), ("data", ctypes.c_void_p), ("len", ctypes.c_size_t),
                ("require_data", ctypes.c_int), ("row_ids", ctypes.POINTER(ctypes.c_uint64)),
                ("rows", ctypes.POINTER(ctypes.c_char_p)), ("row_lens", ctypes.POINTER(ctypes.c_size_t)),
                ("n_rows", ctypes.c_size_t)]


_SIGS = {
    "zg_light_slice_from_slice": (ctypes.c_int, [ctypes.c_char_p, _SZ, ctypes.c_uint32, ctypes.c_uint32,
                                                 ctypes.c_char_p, _SZ, ctypes.POINTER(_SZ)]),
    "zg_light_slice_into_slice": (ctypes.c_int, [ctypes.c_char_p, _SZ, ctypes.c_char_p, _SZ, ctypes.c_uint32,
                                                 ctypes.c_uint32, ctypes.c_char_p, _SZ, ctypes.POINTER(_SZ)]),
    "zg_ctx_msm": (ctypes.c_int, [_P, ctypes.c_uint32, ctypes.c_uint32, _P, _SZ, _P, _P]),
    "zg_submit": (ctypes.c_int, [_P, ctypes.POINTER(_Request), ctypes.POINTER(ctypes.c_uint64)]),
    "zg_wait": (ctypes.c_int, [_P, ctypes.c_uint64, ctypes.c_int64, ctypes.POINTER(_P)]),
    "zg_reply_payload": (_P, [_P, ctypes.POINTER(_SZ)]),
    "zg_encode_batch": (ctypes.c_int, [_P, _SZ, ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(_SZ), ctypes.c_int,
                                       ctypes.POINTER(_P)]),
    "zg_ctx_create": (ctypes.c_int, [ctypes.POINTER(_Config), ctypes.POINTER(_P)]),
    "zg_verify_slices": (ctypes.c_int, [_P, ctypes.POINTER(ctypes.c_char_p), ctypes.POINTER(_SZ), _SZ,
                                        ctypes.c_char_p, ctypes.c_char_p, ctypes.c_uint64,
                                        ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int64)]),
    "zg_ctx_set_pipeline": (ctypes.c_int, [_P, ctypes.POINTER(_PipelineConfig)]),
    "zg_ctx_pipeline_stats": (ctypes.c_int, [_P, ctypes.POINTER(_PipelineStats)]),
    "zg_ctx_autotune": (ctypes.c_int, [_P, ctypes.POINTER(_Tuning)]),
    "zg_ctx_get_tuning": (ctypes.c_int, [_P, ctypes.POINTER(_Tuning)]),
    "zg_ctx_set_tuning": (ctypes.c_int, [_P, ctypes.POINTER(_Tuning)]),
    "zg_ctx_destroy": (None, [_P]),
    "zg_ctx_warmup": (ctypes.c_int, [_P]),
    "zg_encode": (ctypes.c_int, [_P, ctypes.c_char_p, _SZ, ctypes.c_int, ctypes.POINTER(_P)]),
    "zg_reply_free": (None, [_P]),
    "zg_reply_version": (ctypes.c_uint32, [_P]),
    "zg_reply_erasure_commitment": (_P, [_P, ctypes.POINTER(_SZ)]),
    "zg_reply_storage_root": (_P, [_P, ctypes.POINTER(_SZ)]),
    "zg_reply_encoded_data": (_P, [_P, ctypes.POINTER(_SZ)]),
    "zg_reply_num_slices": (_SZ, [_P]),
    "zg_reply_slice": (_P, [_P, _SZ, ctypes.POINTER(_SZ)]),
    "zg_reply_roots": (_P, [_P, ctypes.POINTER(_SZ)]),
    "zg_encode_device": (ctypes.c_int, [_P, _P, _SZ, _P, ctypes.POINTER(_DeviceBlob)]),
    "zg_ctx_param_points": (ctypes.c_int, [_P, ctypes.c_int, ctypes.c_int, _SZ, _SZ, _P, _SZ]),
    "zg_ctx_set_profiling": (ctypes.c_int, [_P, ctypes.c_int]),
    "zg_ctx_phase_times": (ctypes.c_int, [_P, ctypes.POINTER(ctypes.c_float), ctypes.c_int]),
    "zg_ctx_launches": (ctypes.c_uint64, [_P]),
    "zg_probe_imad": (ctypes.c_int, [ctypes.c_int, ctypes.POINTER(ctypes.c_double)]),
    "zg_probe_products": (ctypes.c_int, [ctypes.c_int, ctypes.c_uint32, ctypes.POINTER(ctypes.c_double)]),
    "zg_recover": (ctypes.c_int, [_P, ctypes.POINTER(ctypes.c_uint64), ctypes.POINTER(ctypes.c_char_p),
                                  ctypes.POINTER(_SZ), _SZ, ctypes.c_char_p, _SZ, ctypes.POINTER(_SZ)]),
    "zg_msm_chunks": (ctypes.c_int, [_P, _P, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, _P, _P]),
    "zg_msm_chunks_noalloc": (ctypes.c_int, [_P, _P, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, _P, _P]),
    "zg_ntt": (ctypes.c_int, [_P, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_int, ctypes.c_uint32, _P]),
    "zg_merkle_roots": (ctypes.c_int, [_P, _SZ, _P, _P]),
    "zg_selftest": (ctypes.c_int, [ctypes.POINTER(ctypes.c_int), ctypes.c_int]),
    "zg_last_error": (ctypes.c_char_p, []),
}
C_ABI_FUNCTIONS = sorted(_SIGS)


def lib(build_if_missing=True):
    """The loaded CUDA library. Raises if it is missing and cannot be built."""
    global _lib
    if _lib is None:
        if build_if_missing:
            _build.build()
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(f"CUDA encoder library missing: {LIB_PATH}")
        L = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in _SIGS.items():
            fn = getattr(L, name)
            fn.restype = res
            fn.argtypes = args
        _lib = L
    return _lib


def _check(rc):
    if rc == ZG_OK:
        return
    msg = lib().zg_last_error().decode(errors="replace")
    if rc == ZG_ERR_TOO_LARGE_BLOB:
        raise TooLargeBlob.from_message(msg)
    if rc == ZG_ERR_RECOVERY:
        raise RecoveryError(msg)
    if rc == ZG_ERR_TIMEOUT:
        raise TimeoutError(msg)
    raise RuntimeError(f"zg_encoder error {rc}: {msg}")


@dataclass(frozen=True)
class Dims:
    """Blob geometry (crates/encoder/src/constants.rs:14-28)."""
    log_row: int = 10
    log_col: int = 10
    coset_n: int = 3

    @property
    def rows(self):
        return 1 << self.log_row

    @property
    def cols(self):
        return 1 << self.log_col

    @property
    def raw_blob_size(self):
        return self.rows * self.cols

    @property
    def rows_encoded(self):
        return self.rows * self.coset_n

    @property
    def encoded_blob_size(self):
        return self.rows_encoded * self.cols

    @property
    def max_blob_size(self):
        return 31 * self.raw_blob_size

    @property
    def max_raw_data_size(self):
        return self.max_blob_size - 4

    @property
    def slice_size(self):
        return 312 + 32 * self.cols + 160 * self.log_row


def probe_imad(device=0):
    """Device integer multiply-add rate, 1e9/s."""
    v = ctypes.c_double()
    _check(lib().zg_probe_imad(device, ctypes.byref(v)))
    return v.value


def probe_products(device=0, kind="hybrid"):
    """Fq products per second (1e9) of one product kind as the MSM bucket
    loop issues them (zg_probe_products)."""
    v = ctypes.c_double()
    _check(lib().zg_probe_products(device, MSM_PRODUCTS.index(kind), ctypes.byref(v)))
    return v.value


def selftest():
    """Mismatch counts of the device arithmetic against its host build."""
    names = ["fq_mul", "fq_mul_f64", "fq_add", "fq_sub", "fr_mul", "fr_roundtrip", "xyzz_dbl", "fq_mul_w28",
             "fr_mul_f64", "fq_inverse", "fr_inverse", "fq_inverse_quad", "quad_add", "quad_dbl"]
    fails = (ctypes.c_int * len(names))()
    _check(lib().zg_selftest(fails, len(names)))
    return dict(zip(names, list(fails)))


class EncoderError(Exception):
    pass


class TooLargeBlob(EncoderError):
    """EncoderError::TooLargeBlob { actual, expected_max }."""

    def __init__(self, actual, expected_max):
        super().__init__(f"TooLargeBlob {{ actual: {actual}, expected_max: {expected_max} }}")
        self.actual = actual
        self.expected_max = expected_max

    @classmethod
    def from_message(cls, msg):
        import re
        m = re.search(r"actual: (\d+), expected_max: (\d+)", msg)
        return cls(int(m.group(1)), int(m.group(2))) if m else cls(-1, -1)

    def __eq__(self, o):
        return isinstance(o, TooLargeBlob) and (self.actual, self.expected_max) == (o.actual, o.expected_max)


class RawData:
    """RawData: payload zero-padded to MAX_BLOB_SIZE with its LE u32 length in
    the last four bytes (crates/encoder/src/raw_data.rs:8-72)."""

    def __init__(self, padded: bytes, dims: Dims):
        self.padded = padded
        self.dims = dims

    @classmethod
    def try_from(cls, value: bytes, dims: Dims = Dims()):
        n = len(value)
        if n > dims.max_raw_data_size:
            raise TooLargeBlob(n, dims.max_raw_data_size)
        buf = bytearray(dims.max_blob_size)
        buf[:n] = value
        buf[dims.max_raw_data_size:] = n.to_bytes(4, "little")
        return cls(bytes(buf), dims)

    def as_bytes(self):
        n = int.from_bytes(self.padded[self.dims.max_raw_data_size:], "little")
        return self.padded[:n]


class ZgEncoderParams:
    """Device-resident encoder params of one GPU (a zg_ctx)."""

    def __init__(self, handle, dims: Dims):
        self._h = handle
        self.dims = dims

    @classmethod
    def from_seed(cls, log_row=10, log_col=10, seed=0, device=0, msm_window_bits=0):
        """Params of a seeded tau, built on the GPU by the reference builder's
        rules (power_tau.rs:54-80, prove_params/generate.rs:139-263)."""
        cfg = _Config(log_row, log_col, seed, None, device, msm_window_bits)
        h = ctypes.c_void_p()
        _check(lib().zg_ctx_create(ctypes.byref(cfg), ctypes.byref(h)))
        return cls(h, Dims(log_row, log_col))

    @classmethod
    def from_dir_mont(cls, params_dir, log_row=10, log_col=10, device=0, msm_window_bits=0):
        """Params from the reference's mont files (amt-prove-coset{c}-mont-*.bin)."""
        cfg = _Config(log_row, log_col, 0, os.fsencode(params_dir), device, msm_window_bits)
        h = ctypes.c_void_p()
        _check(lib().zg_ctx_create(ctypes.byref(cfg), ctypes.byref(h)))
        return cls(h, Dims(log_row, log_col))

    @property
    def handle(self):
        return self._h

    def warmup(self):
        _check(lib().zg_ctx_warmup(self._h))

    def param_line(self, coset, line, first=0, count=None):
        """Points [first, first+count) of a param line, 64 B mont x||y each."""
        if count is None:
            count = self.dims.raw_blob_size - first
        n = count * 64
        buf = ctypes.create_string_buffer(n)
        _check(lib().zg_ctx_param_points(self._h, coset, line, first, count, buf, n))
        return buf.raw

    def autotune(self):
        """Time the kernels' free choices on a synthetic blob and keep the
        fastest (zg_ctx_autotune); returns the choice and the times."""
        t = _Tuning()
        _check(lib().zg_ctx_autotune(self.handle, ctypes.byref(t)))
        return _tuning_dict(t)

    def tuning(self):
        t = _Tuning()
        _check(lib().zg_ctx_get_tuning(self.handle, ctypes.byref(t)))
        return _tuning_dict(t)

    def set_tuning(self, msm_product="hybrid", ntt_cols_per_cta=2, ntt_threads=256, msm_task=64,
                   msm_wide_classes=None):
        """Fix the kernels' free choices (zg_ctx_set_tuning); msm_wide_classes
        None keeps every wide-window class the context holds."""
        cur = self.tuning()
        t = _Tuning()
        t.msm_product = MSM_PRODUCTS.index(msm_product)
        t.msm_task = msm_task
        t.msm_wide_classes = cur["msm_wide_avail"] if msm_wide_classes is None else msm_wide_classes
        t.ntt_cols_per_cta, t.ntt_threads = ntt_cols_per_cta, ntt_threads
        _check(lib().zg_ctx_set_tuning(self.handle, ctypes.byref(t)))

    def set_pipeline(self, max_units=0, blobs_per_launch=0, reserve_mib=0):
        """Settings of the request pipeline (zg_ctx_set_pipeline): at most
        max_units units (0 = as free HBM allows), blobs_per_launch blobs fused
        per unit launch (0 = MAX_FUSED_BLOBS, 1 = none), reserve_mib of device
        memory kept free by admission (0 = 4096)."""
        cfg = _PipelineConfig(max_units, blobs_per_launch, reserve_mib)
        _check(lib().zg_ctx_set_pipeline(self._h, ctypes.byref(cfg)))

    def pipeline_stats(self):
        st = _PipelineStats()
        _check(lib().zg_ctx_pipeline_stats(self._h, ctypes.byref(st)))
        return {"units": st.units, "launches_by_blobs": {k + 1: st.launches[k] for k in range(MAX_FUSED_BLOBS)},
                "max_in_flight": st.max_in_flight, "recoveries": st.recoveries, "unit_bytes": st.unit_bytes}

    def set_profiling(self, enable=True):
        _check(lib().zg_ctx_set_profiling(self._h, 1 if enable else 0))

    def phase_times(self):
        """Last encode's phase durations (ms): rs, merkle, msm, aggregate, slices."""
        ms = (ctypes.c_float * 5)()
        _check(lib().zg_ctx_phase_times(self._h, ms, 5))
        return dict(zip(["rs", "merkle", "msm", "aggregate", "slices"], list(ms)))

    def launches(self):
        return lib().zg_ctx_launches(self._h)

    def close(self):
        if self._h:
            lib().zg_ctx_destroy(self._h)
            self._h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


@dataclass
class EncodeBlobReply:
    """grpc/proto/encoder.proto:16-22."""
    version: int = 0
    erasure_commitment: bytes = b""
    storage_root: bytes = b""
    encoded_data: bytes = b""
    encoded_slice: List[bytes] = field(default_factory=list)


def _read_reply(r):
    """(version, commitment, storage root, encoded data, coset roots, slices)
    copied out of a zg_reply, which is then freed."""
    L = lib()
    try:
        n = ctypes.c_size_t()

        def grab(ptr):
            return ctypes.string_at(ptr, n.value) if n.value else b""

        com = grab(L.zg_reply_erasure_commitment(r, ctypes.byref(n)))
        root = grab(L.zg_reply_storage_root(r, ctypes.byref(n)))
        edata = grab(L.zg_reply_encoded_data(r, ctypes.byref(n)))
        roots = grab(L.zg_reply_roots(r, ctypes.byref(n)))
        ns = L.zg_reply_num_slices(r)
        first = L.zg_reply_slice(r, 0, ctypes.byref(n))
        size = n.value
        slices = [ctypes.string_at(first + i * size, size) for i in range(ns)]
        return L.zg_reply_version(r), com, root, edata, roots, slices
    finally:
        L.zg_reply_free(r)


def _encode_raw(params: ZgEncoderParams, data: bytes, require_data: bool):
    r = ctypes.c_void_p()
    _check(lib().zg_encode(params.handle, data, len(data), 1 if require_data else 0, ctypes.byref(r)))
    return _read_reply(r)


class EncodedBlob:
    """EncodedBlob (crates/encoder/src/encoder/blob.rs:26-62), host copy of the
    device results; slices are the ark-serialized EncodedSlice bytes."""

    def __init__(self, commitment, roots, file_root, data, slices):
        self._commitment = commitment
        self._roots = roots
        self._file_root = file_root
        self._data = data
        self._slices = slices

    @classmethod
    def build(cls, raw: bytes, params: ZgEncoderParams):
        """EncodedBlob::build over RawData::try_from(raw) (raises TooLargeBlob)."""
        _, com, root, edata, roots, slices = _encode_raw(params, raw, True)
        return cls(com, roots, root, edata, slices)

    def get_row(self, index) -> bytes:
        assert index < len(self._slices)
        return self._slices[index]

    def get_affine_commitment(self) -> bytes:
        return self._commitment

    get_commitment = get_affine_commitment

    def get_roots(self):
        return [self._roots[32 * i:32 * (i + 1)] for i in range(3)]

    def get_file_root(self) -> bytes:
        return self._file_root

    def get_data(self) -> bytes:
        return self._data


class RecoveryError(Exception):
    """recover_from_da_slice's Err(String); the message is the reference's text."""


def _unset_bytes(n: int) -> bytes:
    """A bytes object of n > 1 unset bytes, for the one call that fills it: one
    allocation of the result, whose pages the copying threads touch first. (A
    zero-filled buffer and a copy of it are two, and the allocator gives 32 MB back
    to the system or keeps it as the heap happens to lie: 14 or 33 ms for a 1024 x
    1024 payload.)"""
    new = ctypes.pythonapi.PyBytes_FromStringAndSize
    new.restype, new.argtypes = ctypes.py_object, (ctypes.c_char_p, ctypes.c_ssize_t)
    return new(None, n)


def recover_from_da_slice(params: ZgEncoderParams, slices: dict) -> bytes:
    """crates/recovery/src/lib.rs:15-43: {row index: 32-byte-element row bytes}
    -> original payload (raises RecoveryError)."""
    L = lib()
    ids = sorted(slices)
    n = len(ids)
    arr = (ctypes.c_uint64 * n)(*ids)
    bufs = (ctypes.c_char_p * n)(*[slices[i] for i in ids])
    lens = (ctypes.c_size_t * n)(*[len(slices[i]) for i in ids])
    out = _unset_bytes(params.dims.max_raw_data_size)
    out_len = ctypes.c_size_t()
    rc = L.zg_recover(params.handle, arr, bufs, lens, n, out, len(out), ctypes.byref(out_len))
    if rc == ZG_ERR_RECOVERY:
        raise RecoveryError(L.zg_last_error().decode())
    _check(rc)
    return out if out_len.value == len(out) else out[:out_len.value]


class LightEncodedSlice:
    """LightEncodedSlice (crates/encoder/src/encoder/light_slice.rs:11-79) as
    its ark-serialized bytes: an EncodedSlice without the row."""

    def __init__(self, data: bytes, dims: "Dims" = None):
        self.data = data
        self.dims = dims or Dims()

    @classmethod
    def from_slice(cls, slice_bytes: bytes, dims: "Dims" = None):
        d = dims or Dims()
        out = ctypes.create_string_buffer(len(slice_bytes))
        n = ctypes.c_size_t()
        _check(lib().zg_light_slice_from_slice(slice_bytes, len(slice_bytes), d.log_row, d.log_col, out, len(out),
                                               ctypes.byref(n)))
        return cls(out.raw[:n.value], d)

    @property
    def index(self) -> int:
        return int.from_bytes(self.data[:8], "little")

    def into_slice(self, row: bytes) -> bytes:
        d = self.dims
        out = ctypes.create_string_buffer(len(self.data) + 32 * d.cols + 40)
        n = ctypes.c_size_t()
        _check(lib().zg_light_slice_into_slice(self.data, len(self.data), row, len(row), d.log_row, d.log_col,
                                               out, len(out), ctypes.byref(n)))
        return out.raw[:n.value]


# EncodedSlice::verify verdicts (zg_verify_slices; the reference's VerifierError variants)
V_OK = 0
V_AMT_INCORRECT_PROOF = 14
V_DESERIALIZE = 30


def verify_slices(params: ZgEncoderParams, slices, commitment: bytes, storage_root: bytes, seed=0):
    """EncodedSlice::verify (crates/encoder/src/encoder/slice.rs:73-95) for a
    batch of serialized slices of one blob, on the GPU (zg_verify_slices).
    Returns (codes, details): per slice the verdict code and its 4 detail
    fields [AmtProofError, a, b, c]. seed=0 draws the batch coefficients from
    the OS CSPRNG; a nonzero seed makes them reproducible, for tests only (a
    party that knows the seed can craft slices that pass)."""
    n = len(slices)
    ptrs = (ctypes.c_char_p * max(n, 1))(*slices)
    lens = (ctypes.c_size_t * max(n, 1))(*[len(x) for x in slices])
    codes = (ctypes.c_int32 * max(n, 1))()
    det = (ctypes.c_int64 * max(4 * n, 1))()
    _check(lib().zg_verify_slices(params.handle, ptrs, lens, n, commitment, storage_root, seed, codes, det))
    return [codes[i] for i in range(n)], [[det[4 * i + k] for k in range(4)] for i in range(n)]


class EncoderService:
    """EncoderService (grpc/src/service.rs:30-105) over device params."""

    def __init__(self, params: ZgEncoderParams):
        self.params = params

    def process_data(self, data: bytes, require_data: bool) -> EncodeBlobReply:
        version, com, root, edata, _, slices = _encode_raw(self.params, data, require_data)
        return EncodeBlobReply(version, com, root, edata, slices)

    def process_batch(self, payloads, require_data: bool) -> List[EncodeBlobReply]:
        """Many process_data calls through the pipelined path (zg_encode_batch);
        replies are bit-identical to process_data's."""
        n = len(payloads)
        ptrs = (ctypes.c_void_p * n)(*[_addr(p) for p in payloads])
        lens = (ctypes.c_size_t * n)(*[_nbytes(p) for p in payloads])
        outs = (ctypes.c_void_p * n)()
        _check(lib().zg_encode_batch(self.params.handle, n, ptrs, lens, 1 if require_data else 0, outs))
        replies = []
        for i in range(n):
            version, com, root, edata, _, slices = _read_reply(ctypes.c_void_p(outs[i]))
            replies.append(EncodeBlobReply(version, com, root, edata, slices))
        return replies

    def submit(self, data, require_data: bool) -> "Ticket":
        """Queue one encode (zg_submit); `data` is bytes or (pointer, length)."""
        q = _Request()
        q.kind = ZG_REQ_ENCODE
        q.data = _addr(data)
        q.len = _nbytes(data)
        q.require_data = 1 if require_data else 0
        return self._submit(q, (data,))

    def submit_recover(self, slices: dict) -> "Ticket":
        """Queue one recover_from_da_slice (crates/recovery/src/lib.rs:15-43)."""
        ids = sorted(slices)
        n = len(ids)
        arr = (ctypes.c_uint64 * n)(*ids)
        bufs = (ctypes.c_char_p * n)(*[slices[i] for i in ids])
        lens = (ctypes.c_size_t * n)(*[len(slices[i]) for i in ids])
        q = _Request()
        q.kind = ZG_REQ_RECOVER
        q.row_ids = arr
        q.rows = bufs
        q.row_lens = lens
        q.n_rows = n
        return self._submit(q, (slices, arr, bufs, lens))

    def _submit(self, q, keep):
        t = ctypes.c_uint64()
        _check(lib().zg_submit(self.params.handle, ctypes.byref(q), ctypes.byref(t)))
        return Ticket(t.value, q.kind, (q,) + keep)

    def wait(self, ticket: "Ticket", timeout_ms: int = -1):
        """The result of a submitted request: an EncodeBlobReply, or the
        recovered payload bytes; raises the request's error."""
        r = ctypes.c_void_p()
        _check(lib().zg_wait(self.params.handle, ticket.id, timeout_ms, ctypes.byref(r)))
        ticket.refs = None
        if ticket.kind == ZG_REQ_RECOVER:
            n = ctypes.c_size_t()
            try:
                p = lib().zg_reply_payload(r, ctypes.byref(n))
                return ctypes.string_at(p, n.value) if n.value else b""
            finally:
                lib().zg_reply_free(r)
        version, com, root, edata, _, slices = _read_reply(r)
        return EncodeBlobReply(version, com, root, edata, slices)


@dataclass
class Ticket:
    """A submitted request; its input buffers stay referenced until wait()."""
    id: int
    kind: int
    refs: tuple = ()


def _addr(data):
    if isinstance(data, tuple):
        return data[0]
    return ctypes.cast(ctypes.c_char_p(data), ctypes.c_void_p).value if len(data) else None


def _nbytes(data):
    return data[1] if isinstance(data, tuple) else len(data)

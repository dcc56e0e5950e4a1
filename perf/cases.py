"""The work that users of the encoder have it do, as a fixed list of cases.

Every case goes through the package's public entry points: the Python API
(EncoderService, recover_from_da_slice, verify_slices) where a program hands
over host bytes, and the C ABI calls that take device pointers
(zg_encode_device, zg_ctx_msm, zg_ntt, zg_merkle_roots) where the data is
already in HBM. Outputs are bytes and whole numbers, so there is no exact():
two correct builds return the same values.

listed() is the fixed list, draw(rng) one more case of the same ranges.
prepare(case, seed) makes the inputs and hands over the encoder context (the
params of one GPU, which a server builds once and keeps for its lifetime;
here one per blob shape and process), run(state) is one pass, work(case) what
a pass cannot do without.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("0g-da-encoder_b200")

TAU_SEED = 2024
FR_PRODUCT_OPS = 2 * 136  # a 256-bit Montgomery product: 64 + 64 + 8 32-bit multiply-adds, two operations each
_contexts = {}
_streams = []


def listed():
    return [
        # a light node's or a test network's blob: the 64 x 32 setting with a
        # short payload, where launches and latency count
        {"name": "encode_64x32", "op": "encode", "log_row": 6, "log_col": 5, "payload": 1234, "data": True},
        # an ordinary request: a ragged payload in a 128 x 1024 blob, slices
        # only (require_data off), host bytes to host slices
        {"name": "encode_128x1024", "op": "encode", "log_row": 7, "log_col": 10, "payload": 2500001, "data": False},
        # the production blob, full payload, resident in HBM end to end
        {"name": "encode_device_1024x1024", "op": "encode_device", "log_row": 10, "log_col": 10,
         "payload": 31 * (1 << 20) - 4},
        # a burst of requests of uneven payloads through the batching path
        {"name": "batch6_128x1024", "op": "batch", "log_row": 7, "log_col": 10, "count": 6, "data": False},
        # single MSMs over a param line: a small one (one latency-bound call),
        # and the full-length one with the blob's own scalar shape
        {"name": "msm_2p12", "op": "msm", "log_row": 10, "log_col": 10, "log_n": 12, "coset": 0, "line": 10,
         "scalars": "uniform"},
        {"name": "msm_2p20", "op": "msm", "log_row": 10, "log_col": 10, "log_n": 20, "coset": 1, "line": 10,
         "scalars": "uniform"},
        # the three transform shapes of the extension: rows, blocks of a few
        # rows on a coset, and the whole blob's inverse
        {"name": "ntt_1024x2p10", "op": "ntt", "log_n": 10, "batch": 1024, "inverse": False, "coset": 0},
        {"name": "ntt_64x2p14_coset", "op": "ntt", "log_n": 14, "batch": 64, "inverse": False, "coset": 1},
        {"name": "ntt_1x2p20_inverse", "op": "ntt", "log_n": 20, "batch": 1, "inverse": True, "coset": 0},
        # the Merkle tree of a production blob's 3072 encoded rows
        {"name": "merkle_3072x1024", "op": "merkle", "log_per_root": 17},
        # a reader's side: the payload of a production blob from half of its
        # rows, and the check of every slice that a signer was handed
        {"name": "recover_1024x1024", "op": "recover", "log_row": 10, "log_col": 10, "rows": 1536},
        {"name": "verify_1024x1024", "op": "verify", "log_row": 10, "log_col": 10, "slices": 3072},
    ]


def _odd_size(rng, lo, hi):
    """log-uniform in [lo, hi]: ragged sizes over the whole range"""
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    shapes = [(4, 6), (6, 5), (5, 10), (7, 10), (10, 10)]
    op = rng.choice(["encode", "encode", "encode_device", "batch", "msm", "msm", "ntt", "ntt", "merkle", "recover",
                     "verify"])
    if op in ("encode", "encode_device"):
        lr, lc = rng.choice(shapes if op == "encode_device" else shapes[:-1])
        case = {"op": op, "log_row": lr, "log_col": lc, "payload": _odd_size(rng, 1, 31 * (1 << (lr + lc)) - 4)}
        if op == "encode":
            case["data"] = rng.random() < 0.5
        return case
    if op == "batch":
        lr, lc = rng.choice(shapes[:-1])
        return {"op": op, "log_row": lr, "log_col": lc, "count": rng.randint(2, 6), "data": rng.random() < 0.5}
    if op == "msm":
        lr, lc = rng.choice([(7, 10), (10, 10)])
        return {"op": op, "log_row": lr, "log_col": lc, "log_n": rng.randint(lc, lr + lc), "coset": rng.randint(0, 2),
                "line": rng.randint(0, lr + 1), "scalars": rng.choice(["uniform", "blob"])}
    if op == "ntt":
        log_n = rng.randint(5, 19)
        inverse = rng.random() < 0.4
        return {"op": op, "log_n": log_n, "batch": _odd_size(rng, 1, 1 << (20 - log_n)) | 1, "inverse": inverse,
                "coset": 0 if inverse else rng.randint(0, 2)}
    if op == "merkle":
        return {"op": op, "log_per_root": rng.randint(4, 16)}
    lr, lc = rng.choice(shapes[1:])
    rows = 1 << lr
    if op == "recover":
        return {"op": op, "log_row": lr, "log_col": lc, "rows": rng.randint(rows, 3 * rows)}
    return {"op": op, "log_row": lr, "log_col": lc, "slices": rng.randint(16, 3 * rows)}


def _params(case):
    key = (case["log_row"], case["log_col"])
    if key not in _contexts:
        _contexts[key] = pkg.ZgEncoderParams.from_seed(*key, seed=TAU_SEED)
    return _contexts[key]


def _stream():
    """the one stream of a program's calls on device memory"""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _payload(seed, n):
    return np.random.default_rng(seed).integers(0, 256, size=n, dtype=np.uint8).tobytes()


def _fr_elements(seed, n, zero_tail=0):
    """n canonical field elements in HBM, uniform below 2^253; the last
    zero_tail of them zero, as in a partly filled blob"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(0, 256, (n, 32), dtype=torch.uint8, device="cuda", generator=g)
    x[:, 31] &= 0x1f
    if zero_tail:
        x[n - zero_tail:] = 0
    return x


def prepare(case, seed):
    op = case["op"]
    state = {"op": op, "case": case}
    if op in ("encode", "batch", "recover", "verify"):
        params = state["params"] = _params(case)
        state["service"] = service = pkg.EncoderService(params)
        dims = params.dims
        if op == "encode":
            state["payload"] = _payload(seed, case["payload"])
        elif op == "batch":
            # ragged lengths up to the largest payload, the same ones for every
            # seed in another order
            sizes = [dims.max_raw_data_size * (i + 1) // case["count"] - 3 * i for i in range(case["count"])]
            order = np.random.default_rng(seed).permutation(case["count"])
            state["payloads"] = [_payload(seed + 100 + int(i), sizes[i]) for i in order]
        else:
            reply = service.process_data(_payload(seed, dims.max_raw_data_size), op == "recover")
            if op == "recover":
                row = 32 * dims.cols
                ids = np.random.default_rng(seed + 1).permutation(dims.rows_encoded)[:case["rows"]]
                state["rows"] = {int(i): reply.encoded_data[row * i:row * (i + 1)] for i in ids}
            else:
                ids = np.random.default_rng(seed + 1).permutation(dims.rows_encoded)[:case["slices"]]
                state["slices"] = [reply.encoded_slice[i] for i in ids]
                # one slice among them has a damaged Merkle leaf (its last byte)
                at = int(np.random.default_rng(seed + 2).integers(case["slices"]))
                state["slices"][at] = state["slices"][at][:-1] + bytes([state["slices"][at][-1] ^ 1])
                state["commitment"], state["root"] = reply.erasure_commitment, reply.storage_root
        return state
    state["stream"] = _stream()
    state["lib"] = pkg.lib()
    if op == "encode_device":
        state["params"] = _params(case)
        g = torch.Generator(device="cuda").manual_seed(seed)
        # the payload starts on a 16-byte boundary, as allocators give it
        state["payload"] = torch.randint(0, 256, (case["payload"],), dtype=torch.uint8, device="cuda", generator=g)
    elif op == "msm":
        state["params"] = _params(case)
        n = 1 << case["log_n"]
        state["scalars"] = _fr_elements(seed, n, n // 5 if case["scalars"] == "blob" else 0)
        state["out"] = torch.empty(64, dtype=torch.uint8, device="cuda")
    elif op == "ntt":
        state["data"] = _fr_elements(seed, case["batch"] << case["log_n"])
    else:
        state["data"] = _fr_elements(seed, _merkle_items(case))
        state["out"] = torch.empty(96, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return state


def _merkle_items(case):
    return 3 << (case["log_per_root"] + 3)


class _DeviceBytes:
    """A device buffer of the library as torch sees it (no copy)."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (int(ptr), False), "version": 3}


def _device_tensor(ptr, n):
    return torch.as_tensor(_DeviceBytes(ptr, n), device="cuda")


def _check(rc):
    if rc:
        raise RuntimeError(pkg.lib().zg_last_error().decode())


def _reply_arrays(reply):
    out = {"commitment": np.frombuffer(reply.erasure_commitment, np.uint8),
           "root": np.frombuffer(reply.storage_root, np.uint8),
           "slices": np.frombuffer(b"".join(reply.encoded_slice), np.uint8)}
    if reply.encoded_data:
        out["data"] = np.frombuffer(reply.encoded_data, np.uint8)
    return out


def run(state):
    op, case = state["op"], state["case"]
    if op == "encode":
        return _reply_arrays(state["service"].process_data(state["payload"], case["data"]))
    if op == "batch":
        return [_reply_arrays(r) for r in state["service"].process_batch(state["payloads"], case["data"])]
    if op == "recover":
        return np.frombuffer(pkg.recover_from_da_slice(state["params"], state["rows"]), np.uint8)
    if op == "verify":
        codes, details = pkg.verify_slices(state["params"], state["slices"], state["commitment"], state["root"])
        return [np.array(codes, np.int64), np.array(details, np.int64)]
    lib, stream = state["lib"], ctypes.c_void_p(state["stream"].cuda_stream)
    if op == "encode_device":
        params, blob = state["params"], pkg._DeviceBlob()
        _check(lib.zg_encode_device(params.handle, ctypes.c_void_p(state["payload"].data_ptr()),
                                    state["payload"].numel(), stream, ctypes.byref(blob)))
        d = params.dims
        return {"data": _device_tensor(blob.encoded_data, 32 * d.encoded_blob_size),
                "slices": _device_tensor(blob.slices, blob.slice_size * d.rows_encoded),
                "amt": _device_tensor(blob.amt_outputs, 3 * (4 * d.rows - 2) * 64),
                "roots": _device_tensor(blob.roots, 96), "root": _device_tensor(blob.file_root, 32)}
    if op == "msm":
        _check(lib.zg_ctx_msm(state["params"].handle, case["coset"], case["line"],
                              ctypes.c_void_p(state["scalars"].data_ptr()), 1 << case["log_n"],
                              ctypes.c_void_p(state["out"].data_ptr()), stream))
        return state["out"]
    if op == "ntt":
        # in place, as the ABI has it: the next pass transforms this pass's result
        _check(lib.zg_ntt(ctypes.c_void_p(state["data"].data_ptr()), case["log_n"], case["batch"],
                          1 if case["inverse"] else 0, case["coset"], stream))
        return state["data"]
    _check(lib.zg_merkle_roots(ctypes.c_void_p(state["data"].data_ptr()), _merkle_items(case),
                               ctypes.c_void_p(state["out"].data_ptr()), stream))
    return state["out"]


def _ntt_products(log_n, batch):
    return batch * (1 << log_n) * log_n / 2


def _msm_products(n):
    # 16 windows of 16 bits, an affine addition (slope, its square, y, and
    # three for a shared inversion) per point and window
    return 16 * 6 * n


def _encode_work(case):
    lr, lc = case["log_row"], case["log_col"]
    n = 1 << (lr + lc)
    slices = 3 * (1 << lr) * (312 + 32 * (1 << lc) + 160 * lr)
    products = 3 * _ntt_products(lr + lc, 1) + 3 * _msm_products(n) * (lr + 2)
    payload = case.get("payload", 31 * n // 2)
    return {"bytes": payload + slices + 96 * n * bool(case.get("data", True)), "flops": products * FR_PRODUCT_OPS}


def work(case):
    op = case["op"]
    if op in ("encode", "encode_device"):
        return _encode_work(case)
    if op == "batch":
        one = _encode_work(case)
        return {k: v * case["count"] for k, v in one.items()}
    if op == "msm":
        n = 1 << case["log_n"]
        n_used = n - n // 5 if case["scalars"] == "blob" else n
        return {"bytes": 32 * n + 64 * n_used + 64, "flops": _msm_products(n_used) * FR_PRODUCT_OPS}
    if op == "ntt":
        n = case["batch"] << case["log_n"]
        return {"bytes": 64 * n, "flops": _ntt_products(case["log_n"], case["batch"]) * FR_PRODUCT_OPS}
    if op == "merkle":
        items = _merkle_items(case)
        # two Keccak-f per 8-item leaf, one per parent; 24 rounds of about 180
        # 32-bit operations each
        perms = 2 * (items // 8) + items // 8
        return {"bytes": 32 * items + 96, "flops": perms * 24 * 180}
    lr, lc = case["log_row"], case["log_col"]
    n = 1 << (lr + lc)
    if op == "recover":
        # the row transforms of what was received, two of 4 R points per
        # column, and the row transforms of the payload
        products = (case["rows"] << lc) * lc / 2 + 2 * (1 << lc) * _ntt_products(lr + 2, 1) + n * lc / 2
        return {"bytes": (case["rows"] << lc) * 32 + 31 * n, "flops": products * FR_PRODUCT_OPS}
    size = 312 + 32 * (1 << lc) + 160 * lr
    # per slice one row's MSM, lr + 1 points with 128-bit coefficients, and a
    # share of the Merkle path
    products = case["slices"] * (_msm_products(1 << lc) + (2 * lr + 1) * 128 * 8)
    return {"bytes": case["slices"] * size, "flops": products * FR_PRODUCT_OPS}

"""Payloads whose digits repeat: one bucket of a wide unit holds most entries."""
import statistics

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_one_byte_repeated_is_no_slower_than_five_random_payloads(gpu_pkg):
    """A 128 x 1024 blob of one byte repeated puts every entry of a 2^16-point
    unit into one bucket. Listed by the bucket's owner alone such a level took
    6.9 times a random payload's encode; the whole CTA lists it (3.3 times,
    the rest is the one item's own additions)."""
    import ctypes
    import torch
    params = gpu_pkg.ZgEncoderParams.from_seed(7, 10, 3)
    n = params.dims.max_raw_data_size
    stream = torch.cuda.Stream()
    blob = gpu_pkg._DeviceBlob()

    def ms(payload):
        data = torch.from_numpy(payload).cuda()
        torch.cuda.synchronize()
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            rc = gpu_pkg.lib().zg_encode_device(params.handle, ctypes.c_void_p(data.data_ptr()), n,
                                                ctypes.c_void_p(stream.cuda_stream), ctypes.byref(blob))
            b.record(stream)
            torch.cuda.synchronize()
            assert rc == 0, gpu_pkg.lib().zg_last_error()
            times.append(a.elapsed_time(b))
        return statistics.median(times[1:])

    random_ms = ms(np.random.default_rng(5).integers(0, 256, n, dtype=np.uint8))
    repeated_ms = ms(np.full(n, 0x55, np.uint8))
    params.close()
    assert repeated_ms < 5 * random_ms, (random_ms, repeated_ms)

"""Device memory of contexts and of the request pipeline's units."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module", autouse=True)
def loaded(gpu_pkg):
    """The driver's own memory (the module, kernels' local memory) comes with the
    first launches of a process and stays."""
    for log_row, log_col in ((6, 5), (5, 10)):
        params = gpu_pkg.ZgEncoderParams.from_seed(log_row, log_col, 1)
        gpu_pkg.EncoderService(params).process_batch([b"x"] * 3, False)
        params.close()


def test_small_context_is_small(gpu_pkg):
    """A 64 x 32 context with one unit of the pipeline: its tables are 26 MB, its
    buffers a few, and the bucket kernel's scratch has a block for each CTA that
    gets a turn, not for the largest context's segments."""
    free0 = _free()
    params = gpu_pkg.ZgEncoderParams.from_seed(6, 5, 1)
    svc = gpu_pkg.EncoderService(params)
    context = free0 - _free()
    replies = svc.process_batch([b"x" * 100, b"y" * 1000], False)
    both = free0 - _free()
    assert [r.storage_root for r in replies] == [svc.process_data(p, False).storage_root
                                                 for p in (b"x" * 100, b"y" * 1000)]
    params.close()
    assert context < 400 << 20, context
    assert both < 900 << 20, both


def test_units_share_the_bucket_scratch(gpu_pkg):
    """Three units in flight take their own buffers, and one scratch; replies are
    those of single calls whatever unit ran before."""
    params = gpu_pkg.ZgEncoderParams.from_seed(5, 10, 2)
    svc = gpu_pkg.EncoderService(params)
    rng = np.random.default_rng(9)
    cap = params.dims.max_raw_data_size
    payloads = [rng.integers(0, 256, int(n), dtype=np.uint8).tobytes() for n in rng.integers(1, cap + 1, 14)]
    payloads[3] = b"\x55" * cap
    plain = [svc.process_data(p, True) for p in payloads]
    free0 = _free()
    assert svc.process_batch(payloads, True) == plain
    stats = params.pipeline_stats()
    held = free0 - _free()
    scratch = held - stats["units"] * stats["unit_bytes"]
    params.close()
    assert stats["unit_bytes"] < 400 << 20, stats
    assert scratch < 2600 << 20, (held, stats)

"""Sizes at which the kernels' splits have an edge: remainders of tiles and units, the smallest and largest of a
range, addresses with the least alignment that an entry point takes."""

import numpy as np
import pytest
import torch

import tensor_b200 as tb
from oracle import gguf_oracle as oracle

pytestmark = pytest.mark.gpu
FORMATS = ("q8_0", "q4_0", "q4_k", "q6_k")


def dev():
    return torch.device("cuda", 0)


def to_dev(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).to(dev())
    return t if dtype is None else t.to(dtype)


@pytest.fixture(scope="module", autouse=True)
def _no_device_timeouts():
    yield
    assert tb.device_status() == 0


# ---- dequantisation: units of 256 weights, four per warp and step ------------------------------------------------

@pytest.mark.parametrize("offset", [0, 2])
@pytest.mark.parametrize("name", FORMATS)
def test_dequant_partial_units_and_two_byte_alignment(name, offset):
    step = tb.get_format(name).weights
    for n, k in [(1, step), (3, 3 * step), (5, 37 * step), (1031, 7 * step)]:
        raw = oracle.make_weights(name, n, k, seed=n + k)
        buf = torch.zeros(raw.size + 16, dtype=torch.uint8, device=dev())
        buf[offset:offset + raw.size] = to_dev(raw)
        out = torch.full((n, k), float("nan"), device=dev())
        tb.dequantize(buf[offset:offset + raw.size], name, n, k, out=out)
        want = oracle.dequantize(raw, name, n, k)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))

"""Quantise-on-load, every way the range of a group is found (within a warp, over a row, neither), with values that repeat
(quotients halfway between two codes), a constant row and a row far from zero: bit for bit against the oracle's quantiser."""
import numpy as np
import pytest
import torch

from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("K,bits,group", [(128, 4, 32), (224 * 32, 4, 7 * 128), (4224, 3, 0), (2048, 8, 1024), (6144, 2, 2048), (640, 8, 64)])
def test_matches_the_oracle_quantiser(abq, oracle, cuda, K, bits, group, symmetric):
    rng = np.random.default_rng(K + bits)
    N = 37
    w = (rng.integers(-40, 41, size=(N, K)) / 64.0).astype(np.float16)
    w[3] = 0.25
    w[4] = rng.normal(1000, 1, size=K).astype(np.float16)
    w[5] = rng.normal(0, 0.02, size=K).astype(np.float16)
    G = K // group if group else 1
    planes = torch.zeros((bits, N, K // 32), dtype=torch.int32, device="cuda")
    scale = torch.zeros((N, G), dtype=torch.float16, device="cuda")
    zero = torch.zeros((N, G), dtype=torch.uint8, device="cuda")
    abq.quantize_weights_half(dev(w), planes, scale, zero, N, K, bits, group, symmetric)
    torch.cuda.synchronize()
    want_codes, want_scale, want_zero = oracle.quantize_weights_minmax(w, bits, group or None, symmetric)
    assert np.array_equal(scale.cpu().numpy().view(np.uint16), want_scale.reshape(N, G).view(np.uint16))
    assert np.array_equal(zero.cpu().numpy(), want_zero.reshape(N, G))
    assert np.array_equal(oracle.unpack(planes.cpu().numpy().view(np.uint32), False), want_codes)

"""CUDA quantizer / packer through the C ABI against the oracle: bit-exact."""
import glob
import os

import numpy as np
import pytest
import torch

from oracle import w8

pytestmark = pytest.mark.gpu

QUANT_FILES = sorted(glob.glob(os.path.join(os.path.dirname(__file__), "golden", "quant_*.npz")))


def _bits(t):
    return t.view(torch.int16 if t.dtype == torch.float16 else torch.int32)


@pytest.mark.parametrize("path", QUANT_FILES, ids=[os.path.basename(p) for p in QUANT_FILES])
def test_quantizer_matches_reference_golden(path):
    from eet_b200 import EET
    g = np.load(path)
    w = torch.from_numpy(g["w"])
    q, packed, scales = EET.quant_weights(w, torch.int8, True)
    assert not q.is_cuda and q.dtype == torch.int8 and tuple(q.shape) == tuple(w.shape)
    assert torch.equal(q, torch.from_numpy(g["q"]))
    assert torch.equal(_bits(scales), _bits(torch.from_numpy(g["scales"])))
    assert scales.dtype == w.dtype
    assert torch.equal(packed, torch.from_numpy(w8.b200_pack_int8(g["q"])))
    # the two-output form returns [packed, scales]
    p2, s2 = EET.quant_weights(w, torch.int8, False)
    assert torch.equal(p2, packed) and torch.equal(_bits(s2), _bits(scales))
    # reference-packed bytes convert to the same layout
    assert torch.equal(EET.repack_reference_weights(torch.from_numpy(g["ref_packed"])), packed)
    assert torch.equal(EET.unpack_weights(packed), q)
    assert torch.equal(EET.preprocess_weights(q), packed)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(64, 64), (4096, 4096), (4096, 11008), (11008, 4096)])
def test_quantizer_matches_oracle_at_config_sizes(dtype, shape):
    """configs[0]/[1] shapes: seeded W ~ N(0, 0.02^2); the C oracle runs these in well under a second."""
    from eet_b200 import EET
    if dtype == torch.float32 and shape[0] * shape[1] > 4096 * 4096:
        pytest.skip("fp32 input covered at 4096x4096")
    K, N = shape
    gen = torch.Generator().manual_seed(0)
    w = (torch.randn(N, K, generator=gen) * 0.02).to(dtype).t().contiguous()
    q, packed, scales = EET.quant_weights(w, torch.int8, True)
    qo, so = w8.c_symmetric_quantize_int8(w.numpy())
    assert torch.equal(q, torch.from_numpy(qo))
    assert torch.equal(_bits(scales), _bits(torch.from_numpy(so)))
    assert torch.equal(packed, torch.from_numpy(w8.c_b200_pack_int8(qo)))


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("K", [64, 128, 192, 320])
def test_quantizer_at_rounding_boundaries(K, dtype, variant):
    """Quotients on, just below and just above every half-integer, scales at the ends of the range and beyond it
    (denormal, zero, huge, infinite), NaN: bit for bit what the division gives, for odd and even numbers of row tiles."""
    from eet_b200 import EET
    gen = torch.Generator().manual_seed(K)
    N = 128
    w = (torch.randint(-256, 257, (K, N), generator=gen) * 0.5)
    w[0] = torch.where(torch.arange(N) % 2 == 0, 128.0, -128.0)
    w = w.to(dtype)
    ulps = torch.randint(-2, 3, (K, N), generator=gen).to(torch.int16 if dtype == torch.float16 else torch.int32)
    w[1:] = (w[1:].view(ulps.dtype) + ulps[1:]).view(dtype)
    expo = torch.linspace(-14 if dtype == torch.float16 else -120, 8 if dtype == torch.float16 else 110, N).round()
    w = (w.double() * torch.pow(torch.tensor(2.0, dtype=torch.float64), expo)).to(dtype)
    w[:, 3] = 0.0
    w[2, 5], w[3, 7], w[4, 9] = float("nan"), float("inf"), float("-inf")
    w[:, 11] = torch.finfo(dtype).tiny / 4
    q, packed, scales = EET.quant_weights(w, torch.int8, True, variant=variant)
    qo, so = w8.c_symmetric_quantize_int8(w.numpy(), variant=variant)
    assert torch.equal(q, torch.from_numpy(qo))
    assert torch.equal(_bits(scales), _bits(torch.from_numpy(so)))
    assert torch.equal(packed, torch.from_numpy(w8.c_b200_pack_int8(qo)))


def test_variant_127_and_three_d_input():
    from eet_b200 import EET
    gen = torch.Generator().manual_seed(4)
    w = (torch.randn(2, 128, 64, generator=gen) * 0.02).half()
    q, packed, scales = EET.quant_weights(w, torch.int8, True, variant=1)
    assert q.shape == (2, 128, 64) and scales.shape == (2, 64)
    for e in range(2):
        qo, so = w8.c_symmetric_quantize_int8(w[e].numpy(), variant=1)
        assert torch.equal(q[e], torch.from_numpy(qo))
        assert torch.equal(_bits(scales[e]), _bits(torch.from_numpy(so)))
    assert int(q.min()) >= -127


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("offset", [4, 8, 12])
def test_quantizer_scratch_needs_no_more_than_float_alignment(dtype, offset):
    """A scratch that begins anywhere in a larger allocation of the caller: the same bits, its neighbours untouched."""
    from eet_b200 import EET
    from eet_b200._lib import check, lib
    K, N = 192, 320
    w = (torch.randn(K, N, generator=torch.Generator().manual_seed(offset)) * 0.02).to(dtype).cuda()
    packed, scales = EET.quant_weights(w, torch.int8)
    ws = torch.full((N + 8,), -3.0, device="cuda")
    p2, s2 = torch.zeros_like(packed), torch.zeros_like(scales)
    check(lib.eet_quantize_w8(w.data_ptr(), int(dtype == torch.float32), K, N, None, p2.data_ptr(), s2.data_ptr(), 0,
                              ws.data_ptr() + offset, 4 * N, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(p2, packed) and torch.equal(_bits(s2), _bits(scales))
    assert bool((ws[: offset // 4] == -3.0).all()) and bool((ws[offset // 4 + N:] == -3.0).all())


def test_cuda_input_stays_on_device_and_bad_shapes_raise():
    from eet_b200 import EET
    w = torch.randn(64, 128, device="cuda").half()
    packed, scales = EET.quant_weights(w, torch.int8)
    assert packed.is_cuda and scales.is_cuda
    with pytest.raises(RuntimeError, match="multiples of 64"):
        EET.quant_weights(torch.randn(60, 64).half(), torch.int8)

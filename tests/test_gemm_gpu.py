"""W8A16 GEMM through the C ABI against the oracle.

Tolerance (stated by the task): max |err| <= 1e-2 * ||row||_inf against an fp32 dequantize-then-matmul;
additionally the result must sit within a few fp16 ulps of the restatement that mirrors the reference's
rounding (fp16(q*scale) weights, fp32 accumulate, one fp16 rounding)."""
import numpy as np
import pytest
import torch

from oracle import ops, w8

pytestmark = pytest.mark.gpu


def _case(K, N, M, seed=0, wstd=0.02):
    gen = torch.Generator().manual_seed(seed)
    w = (torch.randn(N, K, generator=gen) * wstd).half().t().contiguous()
    x = torch.randn(M, K, generator=gen).half()
    qo, so = w8.c_symmetric_quantize_int8(w.numpy())
    return x, torch.from_numpy(qo), torch.from_numpy(so)


def _run(x, q, s, residual=None):
    from eet_b200 import EET
    packed = EET.preprocess_weights(q).cuda()
    y = EET.gemm_w8a16(x.cuda(), packed, s.cuda(), residual=None if residual is None else residual.cuda())
    torch.cuda.synchronize()
    from eet_b200 import _lib
    assert _lib.device_status() == 0
    return y.cpu()


def _check(y, x, q, s):
    ref = ops.gemm_w8a16_fp32(x, q, s)
    tol = 1e-2 * ref.abs().amax(1, keepdim=True)
    err = (y.double() - ref).abs()
    assert (err <= tol).all(), f"max err {err.max():.4g} vs tol {tol.min():.4g}"
    exact = ops.gemm_w8a16(x, q, s, exact=True).double()
    # both are fp16 roundings of nearly the same fp32 number
    assert ((y.double() - exact).abs() <= 2e-3 * ref.abs().amax(1, keepdim=True) + 1e-3).all()


SHARES, ROW, STREAM_K, TILES, PAIRS = range(5)   # plan[0] of eet_gemm_w8a16_plan


def _plan(M, N, K):
    import ctypes
    from eet_b200._lib import check, lib
    plan = (ctypes.c_int * 5)()
    check(lib.eet_gemm_w8a16_plan(M, N, K, plan))
    return tuple(plan)


@pytest.mark.parametrize("K,N,M,kernels", [
    (4096, 32000, 384, (TILES, PAIRS)),    # stream-K 148 us, tiles 100, pairs 94
    (8192, 22016, 384, (TILES, PAIRS)),    # 172, 134
    (8192, 8192, 384, (TILES,)),           # 66, 50
    (13696, 5120, 384, (TILES,)),          # 67, 55
    (5120, 13696, 256, (TILES,)),          # 50, 39
    (4096, 1536, 512, (STREAM_K,)),        # 17.2, 19.3
    (4096, 4096, 100, (STREAM_K,))])       # 14.5, 17.5
def test_models_choose_the_measured_kernel(K, N, M, kernels):
    assert _plan(M, N, K)[0] in kernels


@pytest.mark.parametrize("K,N,M,kernel", [
    (8192, 22016, 8, SHARES), (8192, 24576, 1, SHARES),   # 30.3 us against 36.2 in two waves of tile rows, 33.3 against 36.5
    (8192, 22016, 12, ROW), (4096, 32000, 8, ROW), (5120, 15360, 8, ROW), (8192, 8192, 8, ROW)])
def test_wide_matrices_of_few_rows_avoid_an_empty_wave(K, N, M, kernel):
    """Through the functional form, which has a way around the dispatch for narrow matrices: right, and (the row kernel adds
    in a fixed order, the equal shares in the order of arrival) from the kernel that the plan names."""
    from eet_b200 import EET
    assert _plan(M, N, K)[0] == kernel
    gen = torch.Generator(device="cuda").manual_seed(M)
    q = torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    s = ((torch.rand(N, generator=gen, device="cuda") + 0.5) * K ** -0.5 / 64).half()
    x = torch.randn(M, K, generator=gen, device="cuda").half()
    r = torch.randn(M, N, generator=gen, device="cuda").half()
    packed = EET.preprocess_weights(q)
    out = EET.gemm_w8a16(x, packed, s, residual=r)
    y = (x.double() @ q.double()) * s.double()
    assert ((out.double() - (y + r.double())).abs() <= 2.0 ** -10 * (y.abs() + (y + r.double()).abs()) + 1e-4).all()
    if kernel == ROW:
        assert torch.equal(EET.gemm_w8a16(x, packed, s, residual=r), out)


@pytest.mark.parametrize("K,N,M", [(4096, 4096, 128), (4096, 4096, 250), (4096, 4096, 40), (4096, 11008, 17), (4096, 12288, 300),
                                   (4096, 4096, 1200), (4096, 4096, 8), (4096, 12288, 16), (4096, 22016, 8), (4096, 192, 100)])
def test_calls_behind_one_another_give_the_same_bits(K, N, M):
    """Six hundred calls that nothing waits between, each kernel beginning beside the last CTAs of the one before it: reads of
    a weight stage that are held up by that kernel's memory traffic must not see the stage's next bytes.  Small whole numbers
    as activations, so every fp32 sum is exact whatever the order of the additions."""
    from eet_b200 import EET, _lib
    gen = torch.Generator(device="cuda").manual_seed(N + M)
    q = torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    s = torch.full((N,), 2.0 ** -10, device="cuda").half()
    x = torch.randint(-4, 5, (M, K), generator=gen, device="cuda").half()
    packed = EET.preprocess_weights(q)
    want = ((x.double() @ q.double()) * 2.0 ** -10).half()
    outs = torch.empty(50, M, N, dtype=torch.float16, device="cuda")
    for _ in range(12):
        for out in outs:
            EET.gemm_w8a16(x, packed, s, out=out)
        assert bool((outs == want).all())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("K,N,M", [(4096, 3968, 40), (4096, 3968, 64), (11008, 3968, 17), (11008, 3968, 33), (1984, 8320, 48)])
def test_stream_k_calls_behind_one_another_give_the_same_bits(K, N, M):
    """The stream-K kernel with tiles of 32 and of 64 tokens, two CTAs an SM and rings that wrap, on shapes that the tiles with the
    weights in tensor memory do not take (the plan is part of the case): six hundred calls that nothing waits between, on exact
    sums, and a scratch that is zero again behind them."""
    from eet_b200 import EET, _lib
    assert _plan(M, N, K)[0] == STREAM_K
    gen = torch.Generator(device="cuda").manual_seed(N + M)
    q = torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    s = torch.full((N,), 2.0 ** -10, device="cuda").half()
    x = torch.randint(-4, 5, (M, K), generator=gen, device="cuda").half()
    packed = EET.preprocess_weights(q)
    want = ((x.double() @ q.double()) * 2.0 ** -10).half()
    outs = torch.empty(50, M, N, dtype=torch.float16, device="cuda")
    for _ in range(12):
        for out in outs:
            EET.gemm_w8a16(x, packed, s, out=out)
        assert bool((outs == want).all())
    assert all(int(ws.view(torch.int32).abs().max()) == 0 for ws in EET._pool.gemm_ws.values())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("K,N,M,two", [(4096, 11008, 32, True), (4096, 11008, 64, True), (11008, 4096, 17, False), (4096, 12288, 64, False)])
def test_stream_k_sums_behind_one_another_are_exact(K, N, M, two):
    """eet_gemm_w8a16_accum as a decode chain of 17 to 64 rows calls it (gate and up in one launch, down, QKV), which takes the
    stream-K kernel whatever the dispatch gives a plain call: six hundred launches that nothing waits between.  Whole numbers:
    twelve products on top of one another stay below 2^24, so every sum is exact whatever the order."""
    from eet_b200 import EET, _lib
    gen = torch.Generator(device="cuda").manual_seed(N + M)
    x = torch.randint(-4, 5, (M, K), generator=gen, device="cuda").half()
    q = [torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8) for _ in range(2 if two else 1)]
    packed = [EET.preprocess_weights(w) for w in q]
    want = [x.double() @ w.double() for w in q]
    assert all(float(w.abs().max()) * 12 < 2 ** 24 for w in want)
    sums = [torch.zeros(50, M, N, device="cuda") for _ in q]
    for rep in range(1, 13):
        for i in range(50):
            EET.gemm_w8a16_accum(x, packed[0], sums[0][i], *((packed[1], sums[1][i]) if two else ()))
        assert all(bool((t.double() == rep * w).all()) for t, w in zip(sums, want))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("epilogue", ["plain", "residual"])
@pytest.mark.parametrize("n,M", [(4096, 3), (4096, 16), (1024, 8), (192, 9), (4096, 40), (4096, 100), (4096, 200), (192, 300)])
def test_output_over_the_activations(n, M, epilogue):
    """out=x: no value of x may be overwritten before every CTA has read it.  Repeated, on a busy queue."""
    from eet_b200 import EET
    gen = torch.Generator(device="cuda").manual_seed(n + M)
    q = torch.randint(-127, 128, (n, n), generator=gen, device="cuda", dtype=torch.int8)
    s = ((torch.rand(n, generator=gen, device="cuda") + 0.5) * n ** -0.5 / 64).half()
    x = torch.randn(M, n, generator=gen, device="cuda").half()
    r = torch.randn(M, n, generator=gen, device="cuda").half()
    packed = EET.preprocess_weights(q)
    y = (x.double() @ q.double()) * s.double()
    want = y + (r.double() if epilogue == "residual" else 0)
    bufs = [x.clone() for _ in range(20)]
    for b in bufs:
        EET.gemm_w8a16(b, packed, s, out=b, residual=r if epilogue == "residual" else None)
    tol = 2.0 ** -10 * (y.abs() + want.abs()) + 1e-4
    assert all(bool(((b.double() - want).abs() <= tol).all()) for b in bufs)


def test_no_second_launch_of_more_clusters_of_three_than_find_room():
    """8192 x 8192 at M = 1200 among others: 44 clusters of three behind a wave of single CTAs run in two turns."""
    for K, N in ((8192, 8192), (8192, 24576), (4096, 12288), (4096, 4096)):
        for M in range(300, 3100, 100):
            kernel, _, whole, left, split = _plan(M, N, K)
            assert not (kernel == TILES and whole > 0 and split == 3 and left > 40)


@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 16])
@pytest.mark.parametrize("KN", [(64, 64), (128, 192), (256, 64), (1024, 320)])
def test_small_shapes(KN, M):
    x, q, s = _case(KN[0], KN[1], M, seed=M)
    _check(_run(x, q, s), x, q, s)


@pytest.mark.parametrize("M", [17, 33, 130])
def test_m_above_16(M):
    x, q, s = _case(256, 192, M, seed=5)
    _check(_run(x, q, s), x, q, s)


def test_config0_single_layer():
    """W[4096,4096] ~ N(0, 0.02^2), X[16,4096] ~ N(0,1)."""
    x, q, s = _case(4096, 4096, 16, seed=0)
    _check(_run(x, q, s), x, q, s)


@pytest.mark.parametrize("KN", [(4096, 11008), (11008, 4096), (4096, 12288)])
@pytest.mark.parametrize("M", [1, 8])
def test_llama7b_projection_shapes(KN, M):
    x, q, s = _case(KN[0], KN[1], M, seed=1)
    _check(_run(x, q, s), x, q, s)


def test_one_hot_rows_return_dequantized_weights_exactly():
    """Size-independent property used at full size: a one-hot activation row k must return
    fp16(q[k, :] * scale) bit for bit - it checks packing, tile addressing and the epilogue."""
    K, N = 4096, 11008
    gen = torch.Generator().manual_seed(2)
    q = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    s = (torch.rand(N, generator=gen) * 1e-3 + 1e-4).half()
    rows = torch.tensor([0, 1, 63, 64, 1000, 2047, 2048, 4095, 17, 3000, 77, 4032, 511, 512, 2500, 3999])
    x = torch.zeros(16, K).half()
    x[torch.arange(16), rows] = 1.0
    y = _run(x, q, s)
    want = (q[rows].float() * s.float()[None]).half()
    assert torch.equal(y, want)


def test_linearity_and_residual_epilogue():
    x, q, s = _case(1024, 512, 8, seed=7)
    y1 = _run(x, q, s)
    y2 = _run((x * 2).half(), q, s)           # exact doubling in fp16 -> doubling of the result
    # (the row kernel adds in a fixed order: bit for bit, but for results in fp16's subnormal range)
    usual = y1.abs() >= 2.0 ** -14
    assert torch.equal(y2.float()[usual], y1.float()[usual] * 2) and (y2.float() - 2 * y1.float()).abs()[~usual].sum() < 1e-3
    r = torch.randn(8, 512).half()
    yr = _run(x, q, s, residual=r)
    # fp16(product) + residual in fp16
    assert torch.equal(yr, (y1.float() + r.float()).half())


@pytest.mark.parametrize("K,N,M", [(4096, 4096, 4), (4096, 4096, 40), (1024, 192, 40), (1024, 192, 200), (4096, 22016, 8)])
def test_repeated_calls_leave_scratch_clean(K, N, M):
    """The row kernel, which leaves the scratch alone, the stream-K kernel, the skinny kernel in groups of rows and on a wide
    matrix: whatever sums a call puts there are zero again behind it."""
    from eet_b200 import EET
    x, q, s = _case(K, N, M, seed=9)
    _check(_run(x, q, s), x, q, s)
    for _ in range(3):
        y = _run(x, q, s)
        assert all(int(ws.view(torch.int32).abs().max()) == 0 for ws in EET._pool.gemm_ws.values())
    _check(y, x, q, s)


@pytest.mark.parametrize("K,N,M", [(100, 64, 1), (128, 100, 1), (4096, 4096, 16), (4096, 4096, 17), (4096, 3968, 40), (1984, 4096, 40),
                                   (4096, 8320, 40), (4096, 4096, 64)])
def test_a_refused_call_stores_nothing(K, N, M):
    """Sizes that are no multiple of 64, and up to 64 rows a call without scratch: refused with a reason, on buffers of the whole
    size, so that a refusal that got lost would show as a stored output and nothing worse."""
    from eet_b200 import _lib
    k, n = (K + 63) // 64 * 64, (N + 63) // 64 * 64
    x, out = torch.zeros(M, k, dtype=torch.float16, device="cuda"), torch.full((M, n), 7.0, dtype=torch.float16, device="cuda")
    w, s = torch.zeros(k, n, dtype=torch.int8, device="cuda"), torch.zeros(n, dtype=torch.float16, device="cuda")
    rc = _lib.lib.eet_gemm_w8a16(x.data_ptr(), w.data_ptr(), s.data_ptr(), out.data_ptr(), M, N, K, None, 0, None, 0,
                                 torch.cuda.current_stream().cuda_stream)
    assert rc != 0 and (b"multiples of 64" if (k, n) != (K, N) else b"workspace") in _lib.lib.eet_last_error()
    assert bool((out == 7.0).all())


def test_empty_and_invalid():
    from eet_b200 import EET, _lib
    x, q, s = _case(64, 64, 1)
    packed = EET.preprocess_weights(q).cuda()
    out = EET.gemm_w8a16(torch.empty(0, 64, device="cuda").half(), packed, s.cuda())
    assert out.shape == (0, 64)
    rc = _lib.lib.eet_gemm_w8a16(1, 1, 1, 1, 1, 64, 100, None, 0, None, 0, None)
    assert rc != 0


@pytest.mark.parametrize("kind", ["plain", "residual", "gate"])
@pytest.mark.parametrize("K,N,M,kernel,whole,split", [
    (64, 128, 65, TILES, True, 1), (320, 384, 97, STREAM_K, False, 0), (1024, 640, 513, TILES, False, 4),
    (4096, 4224, 130, STREAM_K, False, 0), (640, 13696, 999, TILES, True, 1), (2048, 896, 4095, TILES, False, 2),
    (5120, 256, 700, TILES, False, 4), (13696, 5120, 600, TILES, False, 2), (192, 38016, 259, TILES, True, 1),
    (2048, 13696, 700, TILES, True, 2), (2048, 7808, 1100, TILES, True, 3), (5120, 13696, 600, TILES, True, 4),
    (1088, 1280, 2000, TILES, False, 3), (1024, 13696, 2049, PAIRS, False, 0), (1152, 2176, 1813, PAIRS, False, 0),
    (1280, 1152, 3434, PAIRS, False, 0), (960, 12928, 1319, PAIRS, False, 0), (3264, 11392, 4006, PAIRS, False, 0)])
def test_prefill_gemm_tiles(K, N, M, kernel, whole, split, kind):
    """Tiles with a lower half only, token tiles that are no multiple of 32, whole waves, whole waves with the remainder split
    over clusters of 2, 3 and 4 in a second launch, split tiles only, tiles on CTA pairs (several per pair, one wave, no
    upper half), few k-blocks; the plan that puts a shape there is part of the case.  Bound: fp32 sums, one fp16 rounding of
    the product and one of the sum with the residual, 2^-11 each, doubled; the activation's error is its operands' plus its
    own three fp16 steps."""
    from eet_b200 import EET, _lib
    plan = _plan(M, N, K)
    assert plan[0] == kernel and (kernel != TILES or ((plan[2] > 0) == whole and plan[4] == split and (plan[3] > 0) == (split > 1)))
    gen = torch.Generator(device="cuda").manual_seed(M)
    q = torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    s = ((torch.rand(N, generator=gen, device="cuda") + 0.5) * K ** -0.5 / 64).half()
    x = torch.randn(M, K, generator=gen, device="cuda").half()
    other = torch.randn(M, N, generator=gen, device="cuda").half()
    out = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    kw = {"residual": {"residual": other}, "gate": {"gate": other}}.get(kind, {})
    EET.gemm_w8a16(x, EET.preprocess_weights(q), s, out=out[:M], **kw)
    y = (x.double() @ q.double()) * s.double()
    if kind == "gate":
        want = torch.nn.functional.silu(other.double()) * y
        tol = 2.0 ** -10 * (4 * want.abs() + y.abs()) + 1e-4
    else:
        want = y + (other.double() if kind == "residual" else 0)
        tol = 2.0 ** -10 * (y.abs() + want.abs()) + 1e-4
    assert ((out[:M].double() - want).abs() <= tol).all()
    assert bool((out[M] == 7.0).all())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("K,N,M,bn,split,tiles", [
    (2112, 22016, 17, 32, 1, 86), (2112, 11008, 17, 32, 3, 43), (2112, 4096, 17, 32, 6, 16), (4096, 8320, 33, 48, 4, 33),
    (2112, 4096, 161, 48, 2, 64), (4096, 5120, 50, 64, 5, 20), (2112, 5120, 111, 64, 3, 40), (2112, 4096, 129, 80, 4, 32),
    (4096, 22016, 233, 80, 1, 258), (2112, 8320, 90, 96, 4, 33), (11008, 5120, 100, 112, 6, 20), (2112, 22016, 300, 112, 1, 258),
    (4096, 4096, 233, 128, 4, 32), (4096, 12288, 127, 128, 2, 48), (2112, 22016, 385, 144, 1, 258), (5120, 4352, 150, 160, 6, 17),
    (2112, 8320, 700, 176, 1, 132), (11008, 5120, 333, 176, 3, 40), (11008, 5120, 190, 192, 6, 20), (2112, 22016, 190, 192, 1, 86)])
@pytest.mark.parametrize("kind", ["plain", "residual", "gate"])
def test_tiles_with_the_weights_in_tensor_memory(K, N, M, bn, split, tiles, kind):
    """Every token tile from the smallest to the largest, units of one and of two k-blocks and an odd k-block at the end (K =
    2112), clusters of every size that a plan uses, chunks of 8 and of 16 tokens with fewer chunks than ranks, persistent CTAs
    with several tiles, a last channel tile of half height (N = 8320); the plan is part of the case.  Bound: one fp16 rounding
    of the product and one of the sum, 2^-11 each, doubled; the activation's error is its operands' plus its own fp16 steps.
    And the same bits from a second call behind a call on other rows."""
    from eet_b200 import EET, _lib
    assert _lib.lib.eet_gemm_w8a16_weights_in_tmem(M, N, K) == 1
    assert _plan(M, N, K) == (TILES, bn, tiles if split == 1 else 0, 0 if split == 1 else tiles, split)
    gen = torch.Generator(device="cuda").manual_seed(M)
    q = torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    s = ((torch.rand(N, generator=gen, device="cuda") + 0.5) * K ** -0.5 / 64).half()
    x = torch.randn(M, K, generator=gen, device="cuda").half()
    other = torch.randn(M, N, generator=gen, device="cuda").half()
    packed = EET.preprocess_weights(q)
    out = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    kw = {"residual": {"residual": other}, "gate": {"gate": other}}.get(kind, {})
    EET.gemm_w8a16(x, packed, s, out=out[:M], **kw)
    EET.gemm_w8a16(x.flip(0), packed, s, **kw)
    again = EET.gemm_w8a16(x, packed, s, **kw)
    y = (x.double() @ q.double()) * s.double()
    if kind == "gate":
        want = torch.nn.functional.silu(other.double()) * y
        tol = 2.0 ** -10 * (4 * want.abs() + y.abs()) + 1e-4
    else:
        want = y + (other.double() if kind == "residual" else 0)
        tol = 2.0 ** -10 * (y.abs() + want.abs()) + 1e-4
    assert ((out[:M].double() - want).abs() <= tol).all()
    assert torch.equal(out[:M], again) and bool((out[M] == 7.0).all())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("K,N,M,kernel,tiles", [
    (8192, 19200, 17, STREAM_K, 0), (12160, 19968, 23, STREAM_K, 0), (16384, 19968, 17, STREAM_K, 0), (5120, 38016, 17, STREAM_K, 0),
    (4096, 38016, 32, STREAM_K, 0), (8192, 19200, 48, TILES, 75), (8192, 22016, 48, TILES, 86), (8192, 24576, 17, TILES, 96),
    (2048, 38016, 64, TILES, 149), (4096, 51200, 40, TILES, 200), (4096, 64000, 32, TILES, 250)])
def test_wide_matrices_of_17_to_64_rows_take_the_faster_kernel(K, N, M, kernel, tiles):
    """Tiles that would leave many SMs idle, or begin another wave for a few, against stream-K (measured, us: 8192 x 19200, M = 17,
    stream-K 35, tiles 40; 12160 x 19968, M = 23, 51 and 65; 5120 x 38016, M = 17, 43 and 52 to 67; the other way round 8192 x
    22016, M = 48, 47 and 39; 2048 x 38016, M = 64, 29 and 22; 4096 x 64000, M = 32, 66 and 52).  And right: one rounding to fp16,
    doubled."""
    from eet_b200 import EET, _lib
    assert _plan(M, N, K)[0] == kernel and (kernel == STREAM_K or _plan(M, N, K)[2:] == (tiles, 0, 1))
    assert _lib.lib.eet_gemm_w8a16_weights_in_tmem(M, N, K) == (kernel == TILES)
    gen = torch.Generator(device="cuda").manual_seed(M)
    q = torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    s = ((torch.rand(N, generator=gen, device="cuda") + 0.5) * K ** -0.5 / 64).half()
    x = torch.randn(M, K, generator=gen, device="cuda").half()
    out = EET.gemm_w8a16(x, EET.preprocess_weights(q), s)
    for c in range(0, N, 8192):
        y = (x.double() @ q[:, c:c + 8192].double()) * s[c:c + 8192].double()
        assert ((out[:, c:c + 8192].double() - y).abs() <= 2.0 ** -10 * y.abs() + 1e-4).all()
    assert _lib.device_status() == 0


@pytest.mark.parametrize("K,N,M,taken", [
    (4096, 4096, 16, 0), (4096, 4096, 17, 1), (4096, 3968, 40, 0), (1984, 4096, 40, 0), (4096, 4224, 40, 0), (4096, 8320, 40, 1),
    (4096, 4096, 64, 1), (4096, 4096, 100, 0), (4096, 11008, 100, 1), (13696, 5120, 999, 1), (5120, 13696, 999, 0), (4096, 4096, 4096, 0)])
def test_shapes_that_go_to_tensor_memory(K, N, M, taken):
    """Both sides of each line of the rule; and up to 64 rows the entry point still refuses a call without scratch."""
    from eet_b200 import _lib
    assert _lib.lib.eet_gemm_w8a16_weights_in_tmem(M, N, K) == taken
    if M <= 64:
        assert _lib.lib.eet_gemm_w8a16(16, 16, 16, 16, M, N, K, None, 0, None, 0, None) != 0 and b"workspace" in _lib.lib.eet_last_error()


@pytest.mark.parametrize("kind", ["plain", "residual", "gate", "gated", "norm", "norm_gated"])
@pytest.mark.parametrize("K,N,M", [(64, 64, 1), (512, 128, 16), (1088, 64, 9), (1088, 2560, 8), (4096, 4096, 7), (5120, 5120, 3),
                                   (2048, 8192, 13), (5120, 13696, 12), (64, 65536, 2)])
def test_decode_gemm_finished_in_one_launch(K, N, M, kind):
    """Every cluster size (8, 4, 3, 2, 1), fewer tiles than warps, shares that do not divide, both token groups, each
    epilogue; the same bits twice (fixed order of the sums).  Bound: fp32 sums, so one fp16 rounding of the product and
    one of the sum with the residual, 2^-11 each, doubled; the activation's error is its operands' plus its own three
    fp16 steps.  With the norm inside, the sums of squares come from a call that stores the input (a product with a
    residual, as in a decoder layer); the activations are rounded once to fp16, at another place than rmsnorm_kernel
    rounds them: 2^-11 each way and each, over the root of the reduction's length."""
    from eet_b200 import EET, _lib
    from eet_b200._lib import check, lib
    gen = torch.Generator(device="cuda").manual_seed(M)
    w = [torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8) for _ in range(2)]
    s = [((torch.rand(N, generator=gen, device="cuda") + 0.5) * K ** -0.5 / 64).half() for _ in w]
    packed = [EET.preprocess_weights(q) for q in w]
    x = torch.randn(M, K, generator=gen, device="cuda").half()
    other = torch.randn(M, N, generator=gen, device="cuda").half()

    stream = torch.cuda.current_stream().cuda_stream
    gamma = squares = None
    xn = x
    if kind.startswith("norm"):
        # x <- x @ w + x from a small square weight, leaving its sums of squares
        wx = torch.randint(-127, 128, (K, K), generator=gen, device="cuda", dtype=torch.int8)
        sx = torch.full((K,), K ** -0.5 / 64, device="cuda").half()
        h = torch.empty_like(x)
        squares = torch.full((M, K // 64), float("nan"), device="cuda")
        check(lib.eet_gemm_w8a16_row(x.data_ptr(), None, None, 0.0, EET.preprocess_weights(wx).data_ptr(), sx.data_ptr(),
                                     None, None, x.data_ptr(), h.data_ptr(), squares.data_ptr(), M, K, K, stream))
        assert torch.allclose(squares, h.float().view(M, -1, 64).square().sum(-1), rtol=1e-5)
        gamma, x = (1 + 0.1 * torch.randn(K, generator=gen, device="cuda")).half(), h
        xn = torch.empty_like(x)
        check(lib.eet_rmsnorm(x.data_ptr(), gamma.data_ptr(), xn.data_ptr(), M, K, 1e-6, stream))

    def call():
        if kind in ("plain", "residual", "gate"):
            return EET.gemm_w8a16(x, packed[0], s[0], **{"residual": {"residual": other}, "gate": {"gate": other}}.get(kind, {}))
        out = torch.empty(M, N, dtype=torch.float16, device="cuda")
        two = kind.endswith("gated")
        check(lib.eet_gemm_w8a16_row(x.data_ptr(), None if gamma is None else gamma.data_ptr(),
                                     None if gamma is None else squares.data_ptr(), 1e-6, packed[0].data_ptr(),
                                     s[0].data_ptr(), packed[1].data_ptr() if two else None, s[1].data_ptr() if two else None,
                                     None, out.data_ptr(), None, M, N, K, stream))
        return out

    out = call()
    y = [(xn.double() @ q.double()) * sc.double() for q, sc in zip(w, s)]
    # two roundings of each activation, independent: five times their root-mean-square effect on a sum of K products
    flip = 5 * 2.0 ** -11 * (xn.double() ** 2 @ torch.full((K, 1), 74.0 ** 2, device="cuda").double()).sqrt() * s[0].double().amax() \
        if gamma is not None else 0.0
    if kind in ("plain", "residual", "norm"):
        want = y[0] + (other.double() if kind == "residual" else 0)
        tol = 2.0 ** -10 * (y[0].abs() + want.abs()) + 1e-4 + flip
    else:
        g, u = (y[0], y[1]) if kind.endswith("gated") else (other.double(), y[0])
        want = torch.nn.functional.silu(g) * u
        tol = 2.0 ** -10 * (4 * want.abs() + u.abs() + g.abs()) + 1e-4 + flip * (u.abs() + g.abs())
    assert ((out.double() - want).abs() <= tol).all()
    assert torch.equal(call(), out)
    assert _lib.device_status() == 0


def test_accumulate_and_fused_finalize_kernels():
    """The decode-path split of the GEMM: sums from eet_gemm_w8a16_accum (two weights in one launch), finished
    by the generic finalize kernel, by the RMSNorm head and by the SwiGLU kernel - each against the oracle."""
    from eet_b200 import EET
    from eet_b200._lib import check, lib
    stream = torch.cuda.current_stream().cuda_stream
    M, K, N = 8, 512, 1024
    x, q1, s1 = _case(K, N, M, seed=21)
    _, q2, s2 = _case(K, N, M, seed=22)
    xc = x.cuda()
    p1, p2 = EET.preprocess_weights(q1).cuda(), EET.preprocess_weights(q2).cuda()
    s1c, s2c = s1.cuda(), s2.cuda()
    sums1 = torch.zeros(M, N, dtype=torch.float32, device="cuda")
    sums2 = torch.zeros_like(sums1)
    EET.gemm_w8a16_accum(xc, p1, sums1, p2, sums2)
    want1 = x.double() @ q1.double()
    want2 = x.double() @ q2.double()
    assert torch.allclose(sums1.cpu().double(), want1, rtol=1e-5, atol=1e-2)
    assert torch.allclose(sums2.cpu().double(), want2, rtol=1e-5, atol=1e-2)
    # SwiGLU head: gate = fp16(sums1*s1), up = fp16(sums2*s2)
    act = torch.empty(M, N, dtype=torch.float16, device="cuda")
    g_ref, u_ref = (sums1.cpu() * s1.float()).half(), (sums2.cpu() * s2.float()).half()
    check(lib.eet_swiglu_finalize(sums1.data_ptr(), s1c.data_ptr(), sums2.data_ptr(), s2c.data_ptr(), act.data_ptr(),
                                  M, N, stream))
    ref = ops.gated_silu(g_ref, u_ref)
    assert torch.allclose(act.cpu().float(), ref.float(), rtol=2e-3, atol=1e-5)
    assert float(sums1.abs().max()) == 0 and float(sums2.abs().max()) == 0
    # RMSNorm head: h = fp16(sums*s) + residual, xn = rmsnorm(h)
    EET.gemm_w8a16_accum(xc, p1, sums1)
    res = torch.randn(M, N).half()
    gamma = (1 + 0.1 * torch.randn(N)).half()
    h_out = torch.empty(M, N, dtype=torch.float16, device="cuda")
    xn = torch.empty_like(h_out)
    resc, gc = res.cuda(), gamma.cuda()
    h_ref = ops.add_residual((sums1.cpu() * s1.float()).half(), res)
    check(lib.eet_rmsnorm_finalize(sums1.data_ptr(), s1c.data_ptr(), resc.data_ptr(), h_out.data_ptr(), gc.data_ptr(),
                                   xn.data_ptr(), M, N, 1e-6, stream))
    assert torch.equal(h_out.cpu(), h_ref)
    assert torch.allclose(xn.cpu().float(), ops.rmsnorm(h_ref, gamma, 1e-6).float(), rtol=1e-3, atol=1e-3)
    assert float(sums1.abs().max()) == 0
    # without sums it is a plain RMSNorm of `residual`
    check(lib.eet_rmsnorm_finalize(None, None, resc.data_ptr(), None, gc.data_ptr(), xn.data_ptr(), M, N, 1e-6, stream))
    assert torch.allclose(xn.cpu().float(), ops.rmsnorm(res, gamma, 1e-6).float(), rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("KN", [(5120, 15360), (5120, 13696), (13696, 5120), (8192, 24576), (8192, 22016), (22016, 8192)])
def test_baichuan13b_and_llama65b_projection_shapes(KN):
    """configs[3] / configs[4] layer shapes at full size: random activations against the fp32 oracle on the
    decode batch of those configs capped at 16 rows, plus a prefill-sized batch through the tensor-core path
    checked on sampled rows (the full fp32 product would take the CPU minutes)."""
    K, N = KN
    gen = torch.Generator().manual_seed(K + N)
    q = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    s = (torch.rand(N, generator=gen) * 3e-4 + 1e-4).half()
    x = torch.randn(16, K, generator=gen).half()
    _check(_run(x, q, s), x, q, s)
    xl = torch.randn(384, K, generator=gen).half()
    y = _run(xl, q, s)
    rows = torch.tensor([0, 1, 63, 64, 127, 128, 255, 256, 300, 383])
    ref = ops.gemm_w8a16_fp32(xl[rows], q, s)
    assert ((y[rows].double() - ref).abs() <= 1e-2 * ref.abs().amax(1, keepdim=True)).all()


@pytest.mark.parametrize("K,N,M", [(4096, 11008, 65), (4096, 11008, 100), (4096, 12288, 128), (8192, 8192, 80),
                                   (5120, 5120, 384), (8192, 3072, 512), (1088, 6144, 300)])
def test_wide_shapes_repeat_bit_for_bit_and_need_no_scratch(K, N, M):
    """From 65 rows on, shapes with enough 256-channel tiles (whole, or split over clusters): the same bits every time, and no
    scratch.  Narrow ones may sum in global memory; without scratch they run on tiles, and with 40 rows they are refused."""
    from eet_b200._lib import check, lib
    from eet_b200 import EET
    gen = torch.Generator(device="cuda").manual_seed(M)
    q = torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    s = ((torch.rand(N, generator=gen, device="cuda") + 0.5) * K ** -0.5 / 64).half()
    x = torch.randn(M, K, generator=gen, device="cuda").half()
    packed = EET.preprocess_weights(q)
    stream = torch.cuda.current_stream().cuda_stream

    def call(w, n, rows=M):
        out = torch.empty(rows, n, dtype=torch.float16, device="cuda")
        rc = lib.eet_gemm_w8a16(x.data_ptr(), w.data_ptr(), s.data_ptr(), out.data_ptr(), rows, n, K, None, 0, None, 0, stream)
        return rc, out
    rc, first = call(packed, N)
    check(rc)
    y = (x.double() @ q.double()) * s.double()
    assert ((first.double() - y).abs() <= 2.0 ** -10 * y.abs() + 1e-4).all()   # one rounding to fp16, doubled
    for _ in range(8):
        assert torch.equal(call(packed, N)[1], first)
    narrow = EET.preprocess_weights(q[:, :128].contiguous())
    rc, part = call(narrow, 128)
    check(rc)
    assert ((part.double() - y[:, :128]).abs() <= 2.0 ** -10 * y[:, :128].abs() + 1e-4).all()
    for rows in (1, 16, 40, 64):
        assert call(narrow, 128, rows)[0] != 0 and b"workspace" in lib.eet_last_error()


@pytest.mark.parametrize("M", [17, 32, 40, 64, 100, 128, 250, 256, 400, 512])
@pytest.mark.parametrize("KN", [(256, 128), (192, 256), (1024, 384), (4096, 4096)])
def test_stream_k_tensor_core_kernel(KN, M):
    """16 < M <= 512 goes to the stream-K tcgen05 kernel: token tiles of 32 / 64 / 128 with ragged tails,
    strips that end inside a CTA's range (small K) and ranges shorter than a strip (large K)."""
    x, q, s = _case(KN[0], KN[1], M, seed=M + KN[1])
    _check(_run(x, q, s), x, q, s)
    res = torch.randn(M, KN[1], generator=torch.Generator().manual_seed(1)).half()
    y = _run(x, q, s, residual=res)
    # (two runs may round differently in the last fp16 bit: the order of the fp32 atomic adds is not fixed)
    assert torch.allclose(y.float(), ops.add_residual(_run(x, q, s), res).float(), rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("M", [24, 64])
def test_stream_k_accumulate_two_weights_exact_sums(M):
    """eet_gemm_w8a16_accum above 16 rows, gate and up in one launch: integer-valued inputs make the fp32
    sums exact, so they must EQUAL the integer product whatever the order of the atomic adds."""
    from eet_b200 import EET
    K, N = 512, 640
    gen = torch.Generator().manual_seed(M)
    x = torch.randint(-4, 5, (M, K), generator=gen).half()
    q1 = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    q2 = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    sums1 = torch.zeros(M, N, dtype=torch.float32, device="cuda")
    sums2 = torch.zeros_like(sums1)
    p1, p2 = EET.preprocess_weights(q1).cuda(), EET.preprocess_weights(q2).cuda()
    for rep in (1, 2):   # the second launch adds on top of the first
        EET.gemm_w8a16_accum(x.cuda(), p1, sums1, p2, sums2)
        assert torch.equal(sums1.cpu().double(), rep * (x.double() @ q1.double()))
        assert torch.equal(sums2.cpu().double(), rep * (x.double() @ q2.double()))
    from eet_b200 import _lib
    assert _lib.device_status() == 0


@pytest.mark.parametrize("K,N,M", [(4096, 11008, 300), (4096, 11008, 512), (128, 14208, 512), (4096, 4096, 250)])
def test_stream_k_token_tiles_and_strips_exact_sums(K, N, M):
    """eet_gemm_w8a16_accum, which always takes the stream-K kernel here: 256-token tiles (single accumulator buffer), one and
    two of them; 128 x 14208 gives every CTA three one-unit strips, i.e. a third accumulation that has to wait for the
    epilogue of the first; two 128-token tiles.  Whole-number inputs: the sums are exact whatever the order."""
    from eet_b200 import EET, _lib
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randint(-4, 5, (M, K), generator=gen, device="cuda").half()
    q = torch.randint(-128, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)
    sums = torch.zeros(M, N, device="cuda")
    want = x.double() @ q.double()
    for rep in (1, 2):
        EET.gemm_w8a16_accum(x, EET.preprocess_weights(q), sums)
        assert torch.equal(sums.double(), rep * want)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("KNM", [(512, 384, 600), (1024, 640, 1000), (256, 4096, 2048), (4096, 4096, 1024),
                                 (4096, 11008, 300), (4096, 11008, 512), (128, 14208, 512)])
def test_large_m_tensor_core_kernels(KNM):
    """The tile kernel at widths that are and are not multiples of 256; ragged last token tile, residual epilogue."""
    assert _plan(KNM[2], KNM[1], KNM[0])[0] == TILES
    K, N, M = KNM
    x, q, s = _case(K, N, M, seed=K + N + M)
    y = _run(x, q, s)
    rows = torch.tensor([r for r in (0, 1, 127, 128, 255, 256, 511, 512, M - 2, M - 1) if r < M])
    ref = ops.gemm_w8a16_fp32(x[rows], q, s)
    assert ((y[rows].double() - ref).abs() <= 1e-2 * ref.abs().amax(1, keepdim=True)).all()
    exact = ops.gemm_w8a16(x[rows], q, s, exact=True).double()
    assert ((y[rows].double() - exact).abs() <= 2e-3 * ref.abs().amax(1, keepdim=True) + 1e-3).all()
    res = torch.randn(M, N, generator=torch.Generator().manual_seed(2)).half()
    yr = _run(x, q, s, residual=res)
    assert torch.equal(yr[rows], ops.add_residual(y[rows], res[rows]))


@pytest.mark.parametrize("M", [64, 256, 1024, 4096])
@pytest.mark.parametrize("KN", [(4096, 4096), (4096, 11008), (11008, 4096)])
def test_llama7b_projection_shapes_across_the_kernel_regimes(KN, M):
    """configs[1] at its large-M points: the three LLaMA-7B projection shapes at M = 64 and 256 (stream-K
    tcgen05 kernel), 1024 and 4096 (large-tile tcgen05 kernels; K = 11008 walks 172 k-blocks, so every
    shared-memory ring wraps dozens of times).  Sampled rows - every 256-token tile of the output is hit -
    against the fp64 dequantize-then-matmul on the CPU, and ALL elements against an fp32 matmul of the same
    dequantized weights run by torch on the GPU (a consistency check of the rows the CPU did not sample)."""
    K, N = KN
    gen = torch.Generator().manual_seed(K + N + M)
    q = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    s = (torch.rand(N, generator=gen) * 3e-4 + 1e-4).half()
    x = torch.randn(M, K, generator=gen).half()
    y = _run(x, q, s)
    rows = sorted({r for t in range(0, M, 256) for r in (t, t + 127, t + 255) if r < M} | {1, M - 2, M - 1})
    rows = torch.tensor(rows[:: max(1, len(rows) // 24)] + [M - 1])
    ref = ops.gemm_w8a16_fp32(x[rows], q, s)
    tol = 1e-2 * ref.abs().amax(1, keepdim=True)
    assert ((y[rows].double() - ref).abs() <= tol).all()
    w = (q.cuda().float() * s.cuda().float()[None])
    full = x.cuda().float() @ w                       # fp32 (TF32 is off by default for matmul): checker only
    err = (y.cuda().float() - full).abs()
    assert bool((err <= 1e-2 * full.abs().amax(1, keepdim=True)).all()), float(err.max())
    res = torch.randn(M, N, generator=gen).half()
    yr = _run(x, q, s, residual=res)
    assert torch.allclose(yr[rows].float(), ops.add_residual(y[rows], res[rows]).float(), rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("KNM", [(1088, 6144, 300), (832, 8192, 130), (2048, 2560, 700), (4096, 4096, 300), (4096, 4096, 512),
                                 (4096, 11008, 200), (11008, 4096, 700)])
def test_split_k_cluster_tiles(KNM):
    """Shapes with fewer 256 x 256 tiles than SMs (24 to 48 of them): where there are enough k-blocks the k-blocks of a tile
    are split over a cluster of 2, 3 or 4 CTAs whose partial accumulators meet through distributed shared memory
    (the first two, of 17 and 13 k-blocks, run as small whole tiles).  A ragged last token tile (blocks past M are neither sent nor reduced), with and without
    the residual.  Every element against an fp32 matmul of
    the dequantized weights run by torch on the GPU (checker only), sampled rows against the fp64 oracle."""
    K, N, M = KNM
    gen = torch.Generator().manual_seed(K + N + M)
    q = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    s = (torch.rand(N, generator=gen) * 3e-4 + 1e-4).half()
    x = torch.randn(M, K, generator=gen).half()
    y = _run(x, q, s)
    rows = torch.tensor(sorted({0, 1, 31, 32, 63, 64, 95, 127, 128, 129, M // 2, M - 2, M - 1} & set(range(M))))
    ref = ops.gemm_w8a16_fp32(x[rows], q, s)
    assert ((y[rows].double() - ref).abs() <= 1e-2 * ref.abs().amax(1, keepdim=True)).all()
    exact = ops.gemm_w8a16(x[rows], q, s, exact=True).double()
    assert ((y[rows].double() - exact).abs() <= 2e-3 * ref.abs().amax(1, keepdim=True) + 1e-3).all()
    full = x.cuda().float() @ (q.cuda().float() * s.cuda().float()[None])
    err = (y.cuda().float() - full).abs()
    assert bool((err <= 1e-2 * full.abs().amax(1, keepdim=True)).all()), float(err.max())
    res = torch.randn(M, N, generator=gen).half()
    yr = _run(x, q, s, residual=res)
    # the partials are added in rank order: the residual run repeats the plain run bit for bit before the add
    assert torch.equal(yr, ops.add_residual(y, res))


@pytest.mark.parametrize("KNM", [(256, 4096, 2560), (192, 2560, 4000), (1088, 2816, 3400), (4096, 12288, 2304)])
def test_persistent_tiles_in_waves(KNM):
    """More 256 x 256 tiles than SMs, and no multiple of them: persistent CTAs take tiles i, i + G, ... and run
    two to four of them back to back on the same rings, barriers and tensor memory (short and odd k-loops of 4, 3
    and 17 k-blocks, a ragged last token tile, the fused QKV shape of LLaMA-7B); with and without the residual, and
    twice in a row (the kernel is deterministic).  Every element against an fp32 matmul of the dequantized weights
    run by torch on the GPU (checker only), sampled rows against the fp64 oracle."""
    K, N, M = KNM
    gen = torch.Generator().manual_seed(K + N + M)
    q = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    s = (torch.rand(N, generator=gen) * 3e-4 + 1e-4).half()
    x = torch.randn(M, K, generator=gen).half()
    y = _run(x, q, s)
    rows = torch.tensor(sorted({0, 1, 255, 256, 257, 511, 1023, 1024, M // 2, M - 257, M - 2, M - 1} & set(range(M))))
    ref = ops.gemm_w8a16_fp32(x[rows], q, s)
    assert ((y[rows].double() - ref).abs() <= 1e-2 * ref.abs().amax(1, keepdim=True)).all()
    full = x.cuda().float() @ (q.cuda().float() * s.cuda().float()[None])
    err = (y.cuda().float() - full).abs()
    assert bool((err <= 1e-2 * full.abs().amax(1, keepdim=True)).all()), float(err.max())
    del full, err
    assert torch.equal(_run(x, q, s), y)
    res = torch.randn(M, N, generator=gen).half()
    yr = _run(x, q, s, residual=res)
    assert torch.equal(yr, ops.add_residual(y, res))


@pytest.mark.parametrize("KNM", [(256, 384, 8), (256, 384, 100), (1024, 640, 1000), (4096, 4096, 512), (256, 4096, 2560),
                                 (1088, 2816, 3400)])
def test_gated_activation_epilogue(KNM):
    """Epilogue 2: the GEMM is the up projection of a gated FFN and applies gated_silu(gate, .) to its own output,
    in every kernel regime (row kernel, stream-K through the finalize launch, tiles - persistent and split over
    clusters - and CTA pairs in their epilogues), in
    place (the output buffer holds the gate values) and out of place.  Expected: the oracle's gated_silu
    (activation_kernel.cu:106-124) of the gate and of this library's plain GEMM output."""
    from eet_b200 import EET, _lib
    K, N, M = KNM
    gen = torch.Generator().manual_seed(K + N + M)
    q = torch.randint(-128, 128, (K, N), generator=gen, dtype=torch.int8)
    s = (torch.rand(N, generator=gen) * 3e-4 + 1e-4).half()
    x = torch.randn(M, K, generator=gen).half()
    gate = (torch.randn(M, N, generator=gen) * 2).half()
    packed = EET.preprocess_weights(q).cuda()
    xc, sc = x.cuda(), s.cuda()
    up = EET.gemm_w8a16(xc, packed, sc)
    want = ops.gated_silu(gate, up.cpu())
    got = EET.gemm_w8a16(xc, packed, sc, gate=gate.cuda())
    buf = gate.cuda().clone()
    got_inplace = EET.gemm_w8a16(xc, packed, sc, out=buf, gate=buf)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    # (the kernels that sum with atomics may round `up` differently in the last fp16 bit from run to run, and the
    # device's expf may differ from the host's in the last bit before its rounding to fp16)
    tol = dict(rtol=4e-3, atol=4e-3)
    assert torch.allclose(got.cpu().float(), want.float(), **tol)
    assert torch.allclose(got_inplace.cpu().float(), want.float(), **tol)
    assert got_inplace.data_ptr() == buf.data_ptr()

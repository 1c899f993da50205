"""Decode and prefill attention through the C ABI against the oracle.

Tolerance: outputs are fp16 values of magnitude <= ~1 built from fp32 sums in a different order than the
oracle's, with logits rounded to fp16 on both sides: |err| <= 2e-3 + 2e-3*|ref| (about two fp16 ulps)."""
import pytest
import torch

from oracle import ops

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _decode(qkv, kc, vc, step, pad=None, alibi=None, slopes=None, rope=1, splits=0, step_dev=None):
    from eet_b200._lib import check, lib
    B, _, H, D = qkv.shape
    T = kc.shape[2]
    ctx = torch.empty(B, H * D, dtype=torch.float16, device="cuda")
    check(lib.eet_decode_mha(qkv.data_ptr(), None, None, kc.data_ptr(), vc.data_ptr(), ctx.data_ptr(), B, H, D, T, step,
                             None if step_dev is None else step_dev.data_ptr(),
                             None if pad is None else pad.data_ptr(),
                             None if alibi is None else alibi.data_ptr(), 0 if alibi is None else alibi.shape[-1],
                             None if slopes is None else slopes.data_ptr(), rope, 10000.0, splits, _stream()))
    torch.cuda.synchronize()
    return ctx.cpu().view(B, H, D)


def _oracle_decode(qkv, k_hist, v_hist, step, pad, alibi_row, rope):
    q, k, v = qkv[:, 0], qkv[:, 1], qkv[:, 2]
    if rope:
        q, k = ops.rope_neox(q, step - 1), ops.rope_neox(k, step - 1)
    kc, vc = k_hist.clone(), v_hist.clone()
    ctx = ops.decode_attention(q, k, v, kc, vc, step, pad, alibi_row)
    return ctx, kc, vc


def _close(a, b):
    return torch.allclose(a.float(), b.float(), atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("step", [1, 2, 17, 128, 640, 1153])
@pytest.mark.parametrize("splits", [0, 1, 4, 8])
def test_decode_rope(step, splits):
    B, H, D, T = 2, 3, 128, 1160
    gen = torch.Generator().manual_seed(step)
    qkv = torch.randn(B, 3, H, D, generator=gen).half()
    kh = torch.randn(B, H, T, D, generator=gen).half()
    vh = torch.randn(B, H, T, D, generator=gen).half()
    ref, kc_ref, vc_ref = _oracle_decode(qkv, kh, vh, step, None, None, True)
    kc, vc = kh.cuda(), vh.cuda()
    got = _decode(qkv.cuda(), kc, vc, step, splits=splits)
    assert _close(got, ref)
    # the new K (rotated) and V were appended at step-1, nothing else moved
    assert _close(kc.cpu()[:, :, step - 1], kc_ref[:, :, step - 1])
    assert torch.equal(vc.cpu()[:, :, step - 1], vc_ref[:, :, step - 1])
    kc_host = kc.cpu()
    kc_host[:, :, step - 1] = kh[:, :, step - 1]
    assert torch.equal(kc_host, kh)


def _decode_plan(B, H, length):
    import ctypes
    from eet_b200._lib import check, lib
    plan = (ctypes.c_int * 2)()
    check(lib.eet_decode_mha_plan(B, H, length, plan))
    return tuple(plan)


@pytest.mark.parametrize("B,H,length,plan", [
    # us with five CTAs per SM, and with four as its rule would split
    (8, 40, 1000, (2, 5)), (5, 32, 1000, (4, 5)), (18, 40, 500, (1, 5)), (32, 40, 500, (1, 5)),   # 33 / 40, 18 / 20, 35 / 44, 59 / 66
    (8, 32, 1000, (2, 4)), (10, 40, 1000, (1, 4)), (24, 40, 500, (1, 4)), (1, 32, 1000, (8, 4))])  # 27 / 24, 51 / 42, 54 / 46, 9.0 / 7.5
def test_decode_takes_five_ctas_per_sm_where_they_save_a_wave_or_a_split(B, H, length, plan):
    assert _decode_plan(B, H, length) == plan


@pytest.mark.parametrize("B,H,step", [(8, 40, 140), (16, 40, 33), (5, 32, 270)])
def test_decode_with_five_ctas_per_sm(B, H, step):
    D, T = 128, step + 3
    assert _decode_plan(B, H, step)[1] == 5
    gen = torch.Generator().manual_seed(step)
    qkv = torch.randn(B, 3, H, D, generator=gen).half()
    kh = torch.randn(B, H, T, D, generator=gen).half()
    vh = torch.randn(B, H, T, D, generator=gen).half()
    pad = torch.arange(B, dtype=torch.long) % step
    ref, _, vc_ref = _oracle_decode(qkv, kh, vh, step, pad, None, True)
    kc, vc = kh.cuda(), vh.cuda()
    assert _close(_decode(qkv.cuda(), kc, vc, step, pad=pad.view(B, 1).cuda()), ref)
    assert torch.equal(vc.cpu(), vc_ref)


def test_decode_beyond_the_reference_4096_limit():
    B, H, D, T, step = 1, 2, 128, 5000, 4800
    gen = torch.Generator().manual_seed(1)
    qkv = torch.randn(B, 3, H, D, generator=gen).half()
    kh = torch.randn(B, H, T, D, generator=gen).half()
    vh = torch.randn(B, H, T, D, generator=gen).half()
    ref, _, _ = _oracle_decode(qkv, kh, vh, step, None, None, True)
    assert _close(_decode(qkv.cuda(), kh.cuda(), vh.cuda(), step), ref)


@pytest.mark.parametrize("pads", [[0, 17], [5, 0], [40, 39]])
def test_decode_left_padding(pads):
    B, H, D, T, step = 2, 4, 128, 64, 41
    gen = torch.Generator().manual_seed(3)
    qkv = torch.randn(B, 3, H, D, generator=gen).half()
    kh = torch.randn(B, H, T, D, generator=gen).half()
    vh = torch.randn(B, H, T, D, generator=gen).half()
    pad = torch.tensor(pads, dtype=torch.long)
    ref, _, _ = _oracle_decode(qkv, kh, vh, step, pad, None, True)
    got = _decode(qkv.cuda(), kh.cuda(), vh.cuda(), step, pad=pad.view(B, 1).cuda(), splits=2)
    assert _close(got, ref)


@pytest.mark.parametrize("step", [1, 33, 300])
def test_decode_alibi_tensor_and_slopes_forms_agree_with_oracle(step):
    B, H, D, T = 2, 8, 128, 320
    gen = torch.Generator().manual_seed(step)
    qkv = torch.randn(B, 3, H, D, generator=gen).half()
    kh = torch.randn(B, H, T, D, generator=gen).half()
    vh = torch.randn(B, H, T, D, generator=gen).half()
    mask = ops.alibi_mask(H, T).half()
    row = mask[:, step - 1, :step].contiguous()        # what the model passes: alibi_mask[:, -1:, :]
    ref, _, _ = _oracle_decode(qkv, kh, vh, step, None, row, False)
    got_t = _decode(qkv.cuda(), kh.cuda(), vh.cuda(), step, alibi=row.view(H, 1, step).cuda(), rope=0)
    slopes = torch.tensor(ops.alibi_slopes(H), dtype=torch.float32).cuda()
    got_s = _decode(qkv.cuda(), kh.cuda(), vh.cuda(), step, slopes=slopes, rope=0)
    assert _close(got_t, ref)
    assert torch.equal(got_t, got_s)


def test_decode_reads_step_from_device_memory():
    B, H, D, T, step = 2, 2, 128, 96, 50
    gen = torch.Generator().manual_seed(8)
    qkv = torch.randn(B, 3, H, D, generator=gen).half()
    kh = torch.randn(B, H, T, D, generator=gen).half()
    vh = torch.randn(B, H, T, D, generator=gen).half()
    ref, _, _ = _oracle_decode(qkv, kh, vh, step, None, None, True)
    from eet_b200._lib import check, lib
    dev = torch.tensor([step - 1, 7], dtype=torch.int32, device="cuda")
    check(lib.eet_advance_steps(dev.data_ptr(), 1, 1, _stream()))
    got = _decode(qkv.cuda(), kh.cuda(), vh.cuda(), 1, step_dev=dev)   # the host value is ignored
    assert _close(got, ref) and dev.tolist() == [step, 7]


@pytest.mark.parametrize("S", [1, 5, 16, 37, 130])
@pytest.mark.parametrize("mode", ["plain", "pad", "alibi"])
def test_prefill(S, mode):
    from eet_b200._lib import check, lib
    B, H, D, T = 2, 3, 128, 140
    gen = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(B, H, S, D, generator=gen).half() for _ in range(3))
    pad = torch.tensor([0, min(3, S - 1)], dtype=torch.long) if mode == "pad" else None
    alibi = ops.alibi_mask(H, T).half()[:, :S, :S].contiguous() if mode == "alibi" else None
    ref = ops.prefill_attention(q, k, v, pad, alibi)           # [B,H,S,D]
    kc = torch.zeros(B, H, T, D, dtype=torch.float16, device="cuda")
    vc = torch.zeros_like(kc)
    kc[:, :, :S], vc[:, :, :S] = k.cuda(), v.cuda()
    ctx = torch.empty(B, S, H * D, dtype=torch.float16, device="cuda")
    qc = q.cuda()
    pad_c = None if pad is None else pad.cuda()
    alibi_c = None if alibi is None else alibi.cuda()
    check(lib.eet_prefill_mha(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), ctx.data_ptr(), B, S, H, D, T,
                              None if pad_c is None else pad_c.data_ptr(),
                              None if alibi_c is None else alibi_c.data_ptr(), S, _stream()))
    torch.cuda.synchronize()
    got = ctx.cpu().view(B, S, H, D).transpose(1, 2)
    # oracle and kernel both feed fp16 probabilities to P.V, but normalise at different points (the oracle
    # rounds p / sum, the blockwise kernel rounds exp(s - running max) and divides at the end)
    assert torch.allclose(got.float(), ref.float(), atol=4e-3, rtol=4e-3)


@pytest.mark.parametrize("case", [(200, [70, 130], "pad"), (512, [0, 0], "plain"), (300, [0, 0], "alibi"),
                                  (96, [0, 95], "pad"), (128, [0, 0], "plain"), (129, [1, 128], "pad"),
                                  (1024, [0, 0], "plain"), (1000, [0, 300], "pad"), (640, [0, 0], "alibi")])
def test_prefill_long_prompts(case):
    """Prompts of several query tiles (the tcgen05 kernel, 128 x 128 tiles, from 96 tokens on): left padding that
    swallows whole key blocks and whole query tiles (their rows must come out zero), prompts of exactly one tile
    and one token more, the configs[2] prompt length and the 1024 tokens of configs[4] (eight key blocks: both
    rings and both score buffers wrap several times), and ALiBi across tiles."""
    from eet_b200._lib import check, lib
    S, pads, mode = case
    B, H, D, T = 2, 2, 128, max(520, S + 8)
    gen = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(B, H, S, D, generator=gen).half() for _ in range(3))
    pad = torch.tensor(pads, dtype=torch.long) if mode == "pad" else None
    alibi = ops.alibi_mask(H, T).half()[:, :S, :S].contiguous() if mode == "alibi" else None
    ref = ops.prefill_attention(q, k, v, pad, alibi)
    kc = torch.zeros(B, H, T, D, dtype=torch.float16, device="cuda")
    vc = torch.zeros_like(kc)
    kc[:, :, :S], vc[:, :, :S] = k.cuda(), v.cuda()
    ctx = torch.full((B, S, H * D), 7.0, dtype=torch.float16, device="cuda")
    qc = q.cuda()
    pad_c = None if pad is None else pad.cuda()
    alibi_c = None if alibi is None else alibi.cuda()
    check(lib.eet_prefill_mha(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), ctx.data_ptr(), B, S, H, D, T,
                              None if pad_c is None else pad_c.data_ptr(),
                              None if alibi_c is None else alibi_c.data_ptr(), S, _stream()))
    torch.cuda.synchronize()
    got = ctx.cpu().view(B, S, H, D).transpose(1, 2)
    assert torch.allclose(got.float(), ref.float(), atol=4e-3, rtol=4e-3)
    if mode == "pad":
        for b, p_len in enumerate(pads):
            if p_len:
                assert float(got[b, :, :p_len].abs().max()) == 0.0   # rows inside the padding are zeroed


@pytest.mark.parametrize("S,offset", [(96, 0), (97, 1), (129, 3), (191, 6), (255, 7), (320, 2)])
def test_prefill_bias_at_any_alignment(S, offset):
    """An arbitrary bias whose rows start at every even address modulo 16 bytes, odd and even row lengths, NaN above the
    diagonal, and nothing of value around the tensor.  Tolerance as above."""
    from eet_b200._lib import check, lib
    B, H, D = 2, 2, 128
    gen = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(B, H, S, D, generator=gen).half() for _ in range(3))
    bias = (2 * torch.randn(H, S, S, generator=gen)).half()
    bias[torch.triu(torch.ones(S, S, dtype=torch.bool), 1).expand(H, S, S)] = float("nan")
    ref = ops.prefill_attention(q, k, v, None, bias)
    store = torch.full((H * S * S + 16,), float("nan"), dtype=torch.float16, device="cuda")
    at = store[offset: offset + H * S * S]
    at.copy_(bias.view(-1))
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    ctx = torch.empty(B, S, H * D, dtype=torch.float16, device="cuda")
    check(lib.eet_prefill_mha(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), ctx.data_ptr(), B, S, H, D, S, None,
                              at.data_ptr(), S, _stream()))
    got = ctx.cpu().view(B, S, H, D).transpose(1, 2)
    assert torch.allclose(got.float(), ref.float(), atol=4e-3, rtol=4e-3)


def _prefill64(q, k, v, bias):
    """Causal attention of one head in 64 bits, and the same with |v|: the bound of an error that is relative to each product."""
    S = q.shape[0]
    scores = (q.double() @ k.double().t()) * float(torch.tensor(128 ** -0.5).half())
    if bias is not None:
        scores = scores + bias.double()
    scores = scores.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device=q.device), 1), float("-inf"))
    p = torch.softmax(scores, -1)
    return p @ v.double(), p @ v.double().abs()


@pytest.mark.parametrize("S,B,H,mode", [(257, 1, 2, "rising"), (300, 1, 2, "steps"), (383, 1, 2, "lowest"), (1100, 1, 130, "plain"),
                                        (2047, 2, 37, "plain")])
def test_prefill_moving_maximum_and_pair_groups(S, B, H, mode):
    """The softmax keeps an old reference until the maximum has outgrown it by 2^8: scores that rise a little with every block,
    by jumps, and from fp16's lowest value; and more (batch, head) pairs than are worked on at a time (64 MiB of keys and
    values), the last group smaller.  Probabilities and outputs are rounded once to fp16 (2^-11 relative each), scores of a few
    hundred in fp32 move an exponential by less than 1e-4."""
    from eet_b200._lib import check, lib
    D = 128
    gen = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(B, H, S, D, generator=gen, device="cuda").half() for _ in range(3))
    bias = None
    t = torch.arange(S, device="cuda")
    if mode == "rising":
        bias = (0.11 * t).half().expand(H, S, S).contiguous()
    elif mode == "steps":
        bias = (37.0 * (t // 90)).half().expand(H, S, S).contiguous()
    elif mode == "lowest":
        bias = torch.where(t < 200, -65504.0, 0.0).half().expand(H, S, S).contiguous()
    ctx = torch.empty(B, S, H, D, dtype=torch.float16, device="cuda")
    check(lib.eet_prefill_mha(q.data_ptr(), k.data_ptr(), v.data_ptr(), ctx.data_ptr(), B, S, H, D, S, None,
                              None if bias is None else bias.data_ptr(), S, _stream()))
    for b, h in {(0, 0), (0, H // 2), (B - 1, H - 2), (B - 1, H - 1)}:
        ref, size = _prefill64(q[b, h], k[b, h], v[b, h], None if bias is None else bias[h])
        err = (ctx[b, :, h].double() - ref).abs()
        if mode == "lowest":   # -65504 leaves a score 8 bits behind the point: up to 2^-9 in an exponent
            assert bool((err[:200] <= 2 ** -7 * size[:200]).all())
            err, size = err[200:], size[200:]
        assert bool((err <= (2 ** -10 + 1e-4) * size + 2 ** -24).all())


def test_decode_finishes_projection_sums_itself():
    """qkv given as the fp32 sums of the projection GEMM + per-channel scales: same result as the fp16 form,
    and the sums are zero afterwards."""
    from eet_b200._lib import check, lib
    B, H, D, T, step = 2, 3, 128, 64, 33
    gen = torch.Generator().manual_seed(12)
    sums = torch.randn(B, 3 * H * D, generator=gen) * 300
    scale = (torch.rand(3 * H * D, generator=gen) * 4e-3 + 1e-3).half()
    qkv = (sums * scale.float()).half().view(B, 3, H, D)
    kh = torch.randn(B, H, T, D, generator=gen).half()
    vh = torch.randn(B, H, T, D, generator=gen).half()
    ref, kc_ref, _ = _oracle_decode(qkv, kh, vh, step, None, None, True)
    kc, vc, sums_c, scale_c = kh.cuda(), vh.cuda(), sums.cuda(), scale.cuda()
    ctx = torch.empty(B, H * D, dtype=torch.float16, device="cuda")
    check(lib.eet_decode_mha(None, sums_c.data_ptr(), scale_c.data_ptr(), kc.data_ptr(), vc.data_ptr(), ctx.data_ptr(),
                             B, H, D, T, step, None, None, None, 0, None, 1, 10000.0, 4, _stream()))
    torch.cuda.synchronize()
    assert _close(ctx.cpu().view(B, H, D), ref)
    assert _close(kc.cpu()[:, :, step - 1], kc_ref[:, :, step - 1])
    assert float(sums_c.abs().max()) == 0


@pytest.mark.parametrize("B,heads,alibi,pad", [(1, 2, False, False), (3, 2, False, True), (16, 32, False, False), (16, 40, True, False),
                                               (17, 2, True, False), (40, 32, False, True), (8, 64, False, False)])
def test_decode_op_alone_is_the_chain_of_its_kernels(B, heads, alibi, pad):
    """The op's call of its own (one call into the library) against the kernels called one by one, three steps: 64 heads are wide
    enough for scratch below 16 rows, 17 and 40 rows need it.  Same kernels, same order; only sums that meet in the order of
    arrival (2 heads, 17 rows; 64 heads) may round the last bit of a projection differently."""
    from eet_b200 import EET
    from eet_b200._lib import check, lib
    h, D, T, hist = heads * 128, 128, 80, 37
    gen = torch.Generator(device="cuda").manual_seed(B)

    def mat(K, N):
        return (EET.preprocess_weights(torch.randint(-127, 128, (K, N), generator=gen, device="cuda", dtype=torch.int8)),
                ((torch.rand(N, generator=gen, device="cuda") + 0.5) * K ** -0.5 / 64).half())

    (w0, s0), (w1, s1) = mat(h, 3 * h), mat(h, h)
    ln = (1 + 0.1 * torch.randn(h, generator=gen, device="cuda")).half()
    none = torch.empty(0)
    desc = EET.MetaDesc(torch.float16, B, heads, h, 1, hist, T, "silu", D, 4 * h, "cuda:0", False, 1e-6, True)
    op = (EET.BaichuanMmha if alibi else EET.LlamaMmha)(desc, w0, s0, none, none, none, w1, s1, none, ln, none)
    op.k_cache[:, :, :hist] = torch.randn(B, heads, hist, D, generator=gen, device="cuda").half()
    op.v_cache[:, :, :hist] = torch.randn(B, heads, hist, D, generator=gen, device="cuda").half()
    kc, vc = op.k_cache.clone(), op.v_cache.clone()
    op.step_ = hist
    pads = (torch.arange(B, device="cuda") % 7).view(B, 1) if pad else none
    for step in range(hist + 1, hist + 4):
        x = torch.randn(B, 1, h, generator=gen, device="cuda").half()
        bias = ops.alibi_mask(heads, T).half()[:, step - 1: step, :step].contiguous().cuda() if alibi else none
        got = op.forward(x, pads, none, True, True, False, bias).clone()
        xn = torch.empty(B, h, dtype=torch.float16, device="cuda")
        check(lib.eet_rmsnorm(x.data_ptr(), ln.data_ptr(), xn.data_ptr(), B, h, 1e-6, _stream()))
        qkv = EET.gemm_w8a16(xn, w0, s0).view(B, 3, heads, D)
        ctx = torch.empty(B, h, dtype=torch.float16, device="cuda")
        check(lib.eet_decode_mha(qkv.data_ptr(), None, None, kc.data_ptr(), vc.data_ptr(), ctx.data_ptr(), B, heads, D, T, step, None,
                                 pads.data_ptr() if pad else None, bias.data_ptr() if alibi else None, step if alibi else 0, None,
                                 0 if alibi else 1, 10000.0, 0, _stream()))
        want = EET.gemm_w8a16(ctx, w1, s1, residual=x.view(B, h)).view(B, 1, h)
        if (B > 16 and heads == 2) or heads == 64:
            assert _close(got, want) and _close(op.k_cache, kc) and _close(op.v_cache, vc)
        else:
            assert torch.equal(got, want) and torch.equal(op.k_cache, kc) and torch.equal(op.v_cache, vc)
    assert op.step_ == hist + 3

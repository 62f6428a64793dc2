"""Model numerics against plain PyTorch fp32 and end-to-end serving of the models."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch

    assert torch.cuda.is_available()
    torch.cuda.set_device(0)
    return torch


def test_nn_layers_match_pytorch(torch_cuda):
    torch = torch_cuda
    from splitrpc_b200 import ops

    F = torch.nn.functional
    x = torch.randn(3, 56, 56, 64, device="cuda").bfloat16()
    ref = F.max_pool2d(x.float().permute(0, 3, 1, 2), 3, 2, 1).permute(0, 2, 3, 1)
    assert torch.equal(ops.maxpool3x3s2(x).float(), ref)
    y = torch.randn(4, 7, 7, 2048, device="cuda").bfloat16()
    torch.testing.assert_close(ops.global_avgpool(y).float(), y.float().mean((1, 2)), rtol=1e-2, atol=1e-2)
    x = torch.randn(2, 13, 9, 72, device="cuda").bfloat16()  # odd sizes: clamped windows on every border
    ref = F.max_pool2d(x.float().permute(0, 3, 1, 2), 3, 2, 1).permute(0, 2, 3, 1)
    assert torch.equal(ops.maxpool3x3s2(x).float(), ref)
    y = torch.randn(3, 5, 5, 640, device="cuda").bfloat16()
    torch.testing.assert_close(ops.global_avgpool(y).float(), y.float().mean((1, 2)), rtol=1e-2, atol=1e-2)
    for m_rows, n_cols, k in ((64, 1000, 2048), (5, 10, 512), (130, 77, 256), (70, 100, 1024)):
        a = torch.randn(m_rows, k, device="cuda").bfloat16()
        w = (torch.randn(n_cols, k, device="cuda") * 0.05).bfloat16()
        bias = torch.randn(n_cols, device="cuda")
        torch.testing.assert_close(ops.fc_skinny(a, w, bias=bias), a.float() @ w.float().t() + bias, rtol=1e-3, atol=1e-3)
    h = torch.randn(300, 768, device="cuda").bfloat16()
    r = torch.randn(300, 768, device="cuda").bfloat16()
    g, b = torch.randn(768, device="cuda"), torch.randn(768, device="cuda")
    ln = ops.layernorm(h, g, b, residual=r)
    torch.testing.assert_close(ln.float(), F.layer_norm(h.float() + r.float(), (768,), g, b, 1e-12), rtol=2e-2, atol=2e-2)
    logits = torch.randn(5, 1000, device="cuda")
    out = torch.zeros(5, 1001, device="cuda")
    ops.softmax_response(logits, 5, out=out, resp_stride=1001 * 4, write_argmax=True)
    torch.cuda.synchronize()
    torch.testing.assert_close(out[:, :1000], torch.softmax(logits, -1), rtol=1e-4, atol=1e-6)
    assert torch.equal(out[:, 1000].view(torch.int32), logits.argmax(-1).int())
    img = torch.randn(2, 3, 224, 224, device="cuda")
    col = torch.zeros(2 * 112 * 112, 192, dtype=torch.bfloat16, device="cuda")
    ops.stem_im2col(col, 2, x=img, mean=(0.1, 0.2, 0.3), inv_std=(2.0, 3.0, 4.0))
    m = torch.tensor([0.1, 0.2, 0.3], device="cuda").view(1, 3, 1, 1)
    s = torch.tensor([2.0, 3.0, 4.0], device="cuda").view(1, 3, 1, 1)
    unf = F.unfold((img - m) * s, 7, padding=3, stride=2).transpose(1, 2).reshape(-1, 3, 7, 7)  # [pix, c, ky, kx]
    got = col[:, :168].float().view(-1, 7, 3, 8)  # [pix, ky, c, kx8]
    torch.testing.assert_close(got[..., :7], unf.permute(0, 2, 1, 3).bfloat16().float(), rtol=0, atol=0)
    assert got[..., 7].abs().max() == 0 and col[:, 168:].abs().max() == 0


@pytest.mark.parametrize("m_rows", [1, 16, 32, 33, 64, 65, 130])
@pytest.mark.parametrize("n_cols,k", [(8, 8), (1000, 24), (1184, 520), (1192, 512), (4100, 2048), (1200, 3616), (1200, 3624), (77, 6400)])
def test_fc_skinny_forms(torch_cuda, m_rows, n_cols, k):
    """Two and four rows per thread, one and two blocks per SM: around 32 and 64 rows, around one block per SM (148 x 8 columns),
    around the K whose weights fit an SM twice (3616), and K that leave some of a row's sixteen threads without a slice."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(m_rows * n_cols + k)
    a = torch.randn(m_rows, k + 8, device="cuda", generator=g).bfloat16()[:, :k]
    w = torch.randn(n_cols, k + 16, device="cuda", generator=g).bfloat16()[:, :k]
    bias = torch.randn(n_cols, device="cuda", generator=g)
    out = torch.full((m_rows + 1, n_cols + 3), 7.0, device="cuda")
    ops.fc_skinny(a, w, bias=bias, out=out[:m_rows, :n_cols])
    want = a.double() @ w.double().t() + bias.double()
    # k products and a bias in fp32, whatever the order: fewer than k + 8 roundings of partial sums
    bound = (a.double().abs() @ w.double().abs().t() + bias.double().abs()) * ((k + 8) * 2.0 ** -24)
    assert bool(((out[:m_rows, :n_cols].double() - want).abs() <= bound).all())
    assert bool((out[m_rows] == 7).all()) and bool((out[:, n_cols:] == 7).all())


@pytest.mark.parametrize("m_rows", [1, 31, 33, 64, 70])
@pytest.mark.parametrize("n_cols,k", [(1, 1544), (127, 1600), (129, 1792), (1000, 2040), (300, 2048)])
def test_fc_on_clusters(torch_cuda, m_rows, n_cols, k):
    """K just above the dispatch line, with CTAs that get one or no k-block, ragged k-blocks, and one or two phases; ragged rows and columns."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(m_rows * n_cols + k)
    a = torch.randn(m_rows, k + 8, device="cuda", generator=g).bfloat16()[:, :k]
    w = torch.randn(n_cols, k + 16, device="cuda", generator=g).bfloat16()[:, :k]
    bias = torch.randn(n_cols, device="cuda", generator=g)
    out = torch.full((m_rows + 1, n_cols + 3), 7.0, device="cuda")
    ops.fc_skinny(a, w, bias=bias, out=out[:m_rows, :n_cols])
    ops.check_status()
    want = a.double() @ w.double().t() + bias.double()
    # a sum of 16 products is within 2^-22 of the sum of their magnitudes, then eight levels of fp32 additions and the bias
    bound = (a.double().abs() @ w.double().abs().t() + bias.double().abs()) * (40 * 2.0 ** -24)
    assert bool(((out[:m_rows, :n_cols].double() - want).abs() <= bound).all())
    assert bool((out[m_rows] == 7).all()) and bool((out[:, n_cols:] == 7).all())
    # a row's result does not depend on the rows beside it, and rows that share their memory are taken as before
    assert torch.equal(ops.fc_skinny(a[-1:], w, bias=bias)[0], out[m_rows - 1, :n_cols])
    same = ops.fc_skinny(a[:1].expand(3, k), w, bias=bias).double()
    assert bool(((same - want[:1]).abs() <= bound[:1] * (k + 8) / 40).all())


@pytest.mark.parametrize("k", [1544, 1792, 2048])
def test_fc_on_clusters_is_as_close_as_fma_chains(torch_cuda, k):
    """Operands of both signs, one or both of them positive, and nearly equal ones: no further from the exact sums than the chains of
    fp32 FMAs that the layer was computed with (their errors, 8 seeds x 64 x 1000 outputs each)."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    chains = {"both": {1544: 7.47e-8, 1792: 7.73e-8, 2048: 7.93e-8}, "one": {1544: 7.49e-8, 1792: 7.68e-8, 2048: 7.95e-8},
              "none": {1544: 3.51e-8, 1792: 3.30e-8, 2048: 3.16e-8}, "near": {1544: 3.41e-8, 1792: 2.93e-8, 2048: 4.10e-8}}
    for signs, limit in chains.items():
        err = norm = 0.0
        for seed in range(8):
            g = torch.Generator(device="cuda").manual_seed(seed)
            a, w = torch.randn(64, k, device="cuda", generator=g), torch.randn(1000, k, device="cuda", generator=g)
            if signs == "near":
                a, w = 1 + 0.1 * a, 1 + 0.1 * w
            else:
                a, w = a.abs() if signs != "both" else a, (w.abs() if signs == "none" else w) / k ** 0.5
            a, w = a.bfloat16(), w.bfloat16()
            want = a.double() @ w.double().t()
            err += float((ops.fc_skinny(a, w).double() - want).square().sum())
            norm += float(want.square().sum())
        assert (err / norm) ** 0.5 <= limit[k], signs
    ops.check_status()


def test_fc_on_clusters_with_infinities(torch_cuda):
    """Infinities, NaN and sums beyond the range come out as they do from plain fp32 additions."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(2)
    a, w = torch.randn(6, 2048, device="cuda", generator=g), torch.randn(130, 2048, device="cuda", generator=g)
    a[1, 7], a[2, 1900], a[3, 300], a[3, 2000] = float("inf"), float("nan"), float("inf"), float("inf")
    a[4] = 3e38
    w[:, :] = w.abs()
    w[::2, 2000] *= -1
    w[5] = 1
    a, w = a.bfloat16(), w.bfloat16()
    out = ops.fc_skinny(a, w, bias=torch.zeros(130, device="cuda"))
    ops.check_status()
    want = torch.where(a.isinf(), torch.zeros_like(a), a).double() @ w.double().t()
    assert bool(torch.isfinite(out[[0, 5]]).all()) and bool(out[1].eq(float("inf")).all()) and bool(out[2].isnan().all())
    assert bool(out[3, ::2].isnan().all()) and bool(out[3, 1::2].eq(float("inf")).all())  # inf - inf, inf + inf
    assert bool(out[4].eq(float("inf")).all())  # 2048 x 3e38 and more
    assert bool(((out[[0, 5]].double() - want[[0, 5]]).abs() <= want[[0, 5]].abs() * 1e-5 + 1e-3).all())


def test_fc_on_clusters_repeats_itself(torch_cuda):
    """Partial sums that cross between CTAs: launches behind one another on two streams give the bits of launches waited for."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(5)
    sets = [(torch.randn(64, 2048, device="cuda", generator=g).bfloat16(), torch.randn(1000, 2048, device="cuda", generator=g).bfloat16())
            for _ in range(4)]
    want = []
    for a, w in sets:
        want.append(ops.fc_skinny(a, w))
        torch.cuda.synchronize()
    outs = [[torch.empty_like(want[0]) for _ in range(40)] for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for i in range(40):
        for s, mine in zip(streams, outs):
            with torch.cuda.stream(s):
                ops.fc_skinny(*sets[i % 4], out=mine[i])
    torch.cuda.synchronize()
    ops.check_status()
    assert all(torch.equal(mine[i], want[i % 4]) for mine in outs for i in range(40))


@pytest.mark.parametrize("seq", [128, 384])
@pytest.mark.parametrize("exponent", [-120, -126.3, -128, -131])
def test_attention_keeps_subnormal_weights(torch_cuda, seq, exponent):
    """One key far above the others in every row and values that make the others' weights count: weights just above and below
    2^-126 of the row's largest."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    heads, B = 2, 3
    H = heads * 64
    qkv = torch.zeros(B * seq, 3, heads, 64, device="cuda")
    qkv[:, 0, :, 0] = 16
    lead = -exponent * 0.6931471805599453 * 8 / 16  # score / 8 in nats
    best = torch.arange(B, device="cuda") * seq + torch.tensor([0, 40, seq - 1], device="cuda")
    qkv[best, 1, :, 0] = lead
    qkv[:, 2] = torch.rand(B * seq, heads, 64, device="cuda") + 0.5
    qkv[:, 2] *= 2.0 ** 100
    qkv[best, 2] = 0
    qkv = qkv.bfloat16()
    out = ops.attention_tc_qkv(qkv.view(B * seq, 3 * H), B, seq, heads)
    ops.check_status()
    q, k, v = (qkv[:, i].double().view(B, seq, heads, 64).transpose(1, 2) for i in range(3))
    want = (torch.softmax(q @ k.transpose(-1, -2) / 8, -1) @ v).transpose(1, 2).reshape(B * seq, H)
    # a bf16 weight w has a spacing of 2^-133 below 2^-126; the exponent itself is rounded to fp32 (2^-18 near 128)
    w = torch.exp(-torch.tensor(16 * qkv[best[0], 1, 0, 0].item() / 8, dtype=torch.float64)).item()
    rel = max(2.0 ** -8, 2.0 ** -134 / w) + 2.0 ** -8 + 2.0 ** -17
    assert ((out.double() - want).abs() <= rel * want.abs()).all()


def test_space_to_depth_stem_matches_conv2d(torch_cuda):
    """stem_s2d + stem_conv (4x1 taps over overlapping 64-channel windows) against an fp32 7x7/2 convolution."""
    torch = torch_cuda
    import torch.nn.functional as F
    from splitrpc_b200 import ops

    nb = 3
    img = torch.randn(nb, 3, 224, 224, device="cuda")
    w = torch.randn(64, 3, 7, 7, device="cuda") * 0.1
    bias = torch.randn(64, device="cuda")
    mean, inv = (0.1, 0.2, 0.3), (2.0, 3.0, 4.0)
    s2d = torch.full((nb, 115, 115, 16), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.stem_s2d(s2d, nb, x=img, mean=mean, inv_std=inv)
    m = torch.tensor(mean, device="cuda").view(1, 3, 1, 1)
    s = torch.tensor(inv, device="cuda").view(1, 3, 1, 1)
    xn = ((img - m) * s).bfloat16().float()
    pad = F.pad(xn, (3, 3, 3, 3))  # [nb, 3, 230, 230]
    want = torch.zeros(nb, 115, 115, 16, device="cuda")
    for dy in range(2):
        for dx in range(2):
            for c in range(3):
                want[..., dy * 8 + dx * 3 + c] = pad[:, c, dy::2, dx::2]
    torch.testing.assert_close(s2d.float(), want, rtol=0, atol=0)
    out = ops.stem_conv(s2d, ops.stem_weight_s2d(w), nb, bias=bias, act="relu")
    ops.check_status()
    ref = F.relu(F.conv2d(xn, w.bfloat16().float(), bias, 2, 3)).permute(0, 2, 3, 1)
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=3e-2)


@pytest.mark.parametrize("seq,heads", [(128, 12), (384, 16)])
def test_attention_matches_pytorch(torch_cuda, seq, heads):
    torch = torch_cuda
    from splitrpc_b200 import ops

    B, H = 2, heads * 64
    qkv = (torch.randn(B * seq, 3 * H, device="cuda") * 0.5).bfloat16()
    out = ops.attention_d64(qkv, B, seq, heads)
    q, k, v = (t.float().view(B, seq, heads, 64).transpose(1, 2) for t in qkv.split(H, dim=1))
    ref = (torch.softmax(q @ k.transpose(-1, -2) / 8.0, -1) @ v).transpose(1, 2).reshape(B * seq, H)
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("seq,heads", [(128, 12), (384, 16)])
def test_tensor_core_attention_with_v_in_place(torch_cuda, seq, heads):
    """V read in place from the fused Q|K|V buffer (MN-major operand of the second product)."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    B, H = 3, heads * 64
    qkv = (torch.randn(B * seq, 3 * H, device="cuda") * 0.6).bfloat16()
    out = ops.attention_tc_qkv(qkv, B, seq, heads)
    torch.cuda.synchronize()
    ops.check_status()
    q, k, v = (t.float().view(B, seq, heads, 64).transpose(1, 2) for t in qkv.split(H, dim=1))
    ref = (torch.softmax(q @ k.transpose(-1, -2) / 8.0, -1) @ v).transpose(1, 2).reshape(B * seq, H)
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("seq,heads", [(128, 12), (384, 16)])
def test_tensor_core_attention_matches_pytorch(torch_cuda, seq, heads):
    torch = torch_cuda
    from splitrpc_b200 import ops

    B, H = 3, heads * 64
    qk = (torch.randn(B * seq, 2 * H, device="cuda") * 0.7).bfloat16()
    v = (torch.randn(B * seq, H, device="cuda") * 0.5).bfloat16()
    vb = torch.randn(H, device="cuda")
    out = ops.attention_tc(qk, v.t().contiguous(), B, seq, heads, v_bias=vb)
    ops.check_status()
    q, k = (t.float().view(B, seq, heads, 64).transpose(1, 2) for t in qk.split(H, dim=1))
    vv = v.float().view(B, seq, heads, 64).transpose(1, 2)
    ref = (torch.softmax(q @ k.transpose(-1, -2) / 8.0, -1) @ vv).transpose(1, 2).reshape(B * seq, H) + vb
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("fuse_shortcut", [True, False])
def test_resnet50_matches_fp32_reference(torch_cuda, fuse_shortcut):
    torch = torch_cuda
    from splitrpc_b200 import ops
    from splitrpc_b200.models import ResNet50

    n = 16
    m = ResNet50(device=0, max_batch=n, fuse_shortcut=fuse_shortcut)
    x = torch.randn(n, 3, 224, 224, device="cuda")
    out = torch.zeros(n, 1000, device="cuda")
    m.forward(n, x=x, out=out)
    ops.check_status()
    # the oracle in true fp32: no TF32 in cuDNN or cuBLAS
    tf32 = (torch.backends.cudnn.allow_tf32, torch.backends.cuda.matmul.allow_tf32)
    torch.backends.cudnn.allow_tf32 = torch.backends.cuda.matmul.allow_tf32 = False
    try:
        ref = m.reference_forward(x)
    finally:
        torch.backends.cudnn.allow_tf32, torch.backends.cuda.matmul.allow_tf32 = tf32
    assert torch.isfinite(out).all() and (out.sum(1) - 1.0).abs().max().item() < 1e-3
    # bf16 activations through 53 layers: compare the probability rows as vectors
    cos = torch.nn.functional.cosine_similarity(out, ref, dim=1)
    rel = ((out - ref).norm(dim=1) / ref.norm(dim=1)).max().item()
    agree = (out.argmax(1) == ref.argmax(1)).float().mean().item()
    print(f"resnet50 fuse={fuse_shortcut}: min cos {cos.min().item():.5f}, max rel err {rel:.4f}, argmax agreement {agree:.3f}")
    assert cos.min().item() > 0.999, cos  # measured: 0.99999
    assert rel < 0.05, rel                # measured: 0.006 - 0.007
    assert agree >= 15 / 16, agree        # measured: 16 of 16
    # where the oracle is decisive (its best class leads the runner-up by more than the bf16 noise), the classes agree
    top2 = ref.topk(2, dim=1).values
    decisive = (top2[:, 0] - top2[:, 1]) > 0.1 * top2[:, 0]
    assert bool((out.argmax(1) == ref.argmax(1))[decisive].all())


def test_bert_matches_fp32_reference(torch_cuda):
    torch = torch_cuda
    from splitrpc_b200 import ops
    from splitrpc_b200.models import BertClassifier, BERT_BASE

    m = BertClassifier(BERT_BASE, seq=128, device=0, max_batch=4)
    ids = torch.randint(0, 30522, (3, 128), device="cuda", dtype=torch.int32)
    out = torch.zeros(3, 2, device="cuda")
    m.forward(3, ids=ids, out=out)
    ops.check_status()
    ref = m.reference_forward(ids)
    torch.testing.assert_close(out, ref, rtol=5e-2, atol=3e-2)


def test_fused_gather_deserialise_matches_stem_s2d(torch_cuda):
    """The gather that writes normalised space-to-depth tensors into ring slots against stem_s2d on the raw bytes;
    fragments are given out of order and split at odd (4-byte aligned) places."""
    torch = torch_cuda
    from splitrpc_b200 import _C, ops

    n, req = 3, 3 * 224 * 224 * 4
    slot_bytes = req
    img = torch.randn(n, 3, 224, 224, device="cuda")
    raw = img.view(torch.uint8).reshape(n, req)
    ring = torch.zeros(8 * slot_bytes, dtype=torch.uint8, device="cuda")
    mean, inv = (0.1, 0.2, 0.3), (2.0, 3.0, 4.0)
    items = []
    cuts = [0, 8192, 8192 + 4, 100000, 100000 + 16388, 300004, req]
    for r in range(n):
        slot = 2 + r  # the batch sits in slots 2..4
        for a, b in reversed(list(zip(cuts[:-1], cuts[1:]))):
            items.append((raw[r].data_ptr() + a, ring.data_ptr() + slot * slot_bytes + a, b - a))
    h = _C.sg_list_create(items)
    _C.sg_list_launch_stem_s2d(h, ring.data_ptr(), slot_bytes, list(mean), list(inv), -2, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    _C.sg_list_destroy(h)
    want = torch.zeros(n, 115, 115, 16, dtype=torch.bfloat16, device="cuda")
    ops.stem_s2d(want, n, x=img, mean=mean, inv_std=inv)
    torch.cuda.synchronize()
    got = torch.stack([ring[(2 + r) * slot_bytes:(2 + r) * slot_bytes + 115 * 115 * 32].view(torch.bfloat16).view(115, 115, 16)
                       for r in range(n)])
    assert torch.equal(got, want)
    assert int(ring[:2 * slot_bytes].max()) == 0 and int(ring[5 * slot_bytes:].max()) == 0


@pytest.mark.parametrize("fused_ingress", [True, False])
def test_model_server_end_to_end_resnet(torch_cuda, fused_ingress):
    torch = torch_cuda
    from splitrpc_b200.models import ResNet50
    from splitrpc_b200.serving import ModelServer

    m = ResNet50(device=0, max_batch=8)
    srv = ModelServer(m, device=0, max_batch=8, outstanding=16, fused_ingress=fused_ingress)
    assert srv.fused_ingress == fused_ingress
    with srv:
        cli = srv.client(total=48, warmup=0, payload="normal", verify=True, n_payloads=4)
        assert cli.run_closed_loop(16)
        assert cli.received == 48
        stats = srv.server.stats()
        ws = srv.server.worker_stats(0)
    assert stats["sg_errors"] == 0 and ws["wait_timeouts"] == 0
    x = torch.from_numpy(np.frombuffer(cli.payload(1), dtype=np.float32).copy()).view(1, 3, 224, 224).cuda()
    direct = torch.zeros(1, 1000, device="cuda")
    m.forward(1, x=x, out=direct)
    torch.cuda.synchronize()
    got = torch.from_numpy(np.frombuffer(cli.response(5), dtype=np.float32).copy())  # request 5 used payload 5 % 4 == 1
    torch.testing.assert_close(got, direct[0].cpu(), rtol=1e-3, atol=1e-5)


@pytest.mark.parametrize("n", [1, 7, 255, 257, 2047, 2048, 2049, 5000])
def test_softmax_response_lengths(torch_cuda, n):
    """Rows shorter than a block, as long as its registers, longer; rows with -infinity, of one value, with no finite value or a NaN; the
    largest logit in every part of the row."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(12, n + 3, device="cuda", generator=g)[:, :n] * 4
    for r in range(6):
        x[r, (r * (n - 1)) // 5] = 17.0 + r  # the first, the last, and between
    x[6, ::2] = -float("inf")
    x[6, n - 1] = 3.0
    x[7] = -3e38
    x[8] = -float("inf")
    x[9, n // 2] = float("nan")
    x[10] = 0.25
    out = torch.full((13, n + 5), 7.0, device="cuda")
    ops.softmax_response(x, 12, out=out, resp_stride=(n + 5) * 4, write_argmax=True)
    torch.cuda.synchronize()
    want = torch.softmax(x.double(), -1)
    got = out[:12, :n]
    assert torch.equal(got.isnan(), want.isnan())
    # the fast exponential is off by up to 2 + 1.2 |x| units of 2^-23 for differences |x| up to about 40, twice (weight and sum)
    ok = [0, 1, 2, 3, 4, 5, 6, 7, 10, 11]
    assert bool(((got[ok].double() - want[ok]).abs() <= want[ok] * (2 * 50 * 2.0 ** -23) + 1e-37).all())
    arg = out[:12, n].contiguous().view(torch.int32)
    assert [int(a) for a in arg[:6]] == [(r * (n - 1)) // 5 for r in range(6)] and (n < 3 or int(arg[6]) == int(x[6].argmax()))
    assert bool((out[12] == 7).all()) and bool((out[:, n + 1:] == 7).all())


@pytest.mark.parametrize("hidden", [256, 512, 768, 1024])
@pytest.mark.parametrize("rows", [1, 2, 3, 7, 127, 1775, 1777, 2051, 2959, 3949, 7517])
def test_layernorm_rows_per_block(torch_cuda, rows, hidden):
    """Two and four rows per group, one to four groups per block, last blocks with rows or groups missing, residual added or not, rows with a large offset."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    x = (torch.randn(rows, hidden, device="cuda") + 20.0).bfloat16()
    res = torch.randn(rows, hidden, device="cuda").bfloat16()
    g, b = torch.randn(hidden, device="cuda"), torch.randn(hidden, device="cuda")
    buf = torch.full((rows + 1, hidden), 7.0, device="cuda", dtype=torch.bfloat16)
    for r in (None, res):
        ops.layernorm(x, g, b, residual=r, out=buf[:rows])
        xd = x.double() if r is None else x.double() + r.double()
        ref = torch.nn.functional.layer_norm(xd, (hidden,), g.double(), b.double(), 1e-12)
        # bf16 rounding of the result (2^-9 of it), and the fp32 mean and deviations of values about 20 times their spread
        assert ((buf[:rows].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + g.abs().double() * 2e-5 + 1e-6).all()
        assert (buf[rows] == 7.0).all()


@pytest.mark.parametrize("batch,seq,hidden", [(1, 1, 768), (1, 3, 1024), (5, 7, 768), (14, 127, 768), (14, 127, 1024), (32, 127, 768), (24, 127, 1024),
                                              (1, 1, 256), (3, 3, 256), (7, 127, 256), (1, 3, 512), (5, 7, 512), (60, 127, 512)])
def test_embedding_layernorm_tokens_per_block(torch_cuda, batch, seq, hidden):
    """Two and four tokens per group, one to four groups per block, last blocks with tokens or groups missing, groups across sequences, ids
    outside the vocabulary."""
    torch = torch_cuda
    from splitrpc_b200 import ops

    vocab = 50
    word, pos, typ = (torch.randn(n, hidden, device="cuda").bfloat16() for n in (vocab, seq, 2))
    g, b = torch.randn(hidden, device="cuda"), torch.randn(hidden, device="cuda")
    ids = torch.randint(-5, vocab + 5, (batch, seq), device="cuda", dtype=torch.int32)
    buf = torch.full((batch * seq + 1, hidden), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.bert_embed_ln(buf[: batch * seq], batch, seq, word, pos, typ, g, b, ids=ids)
    x = word.double()[ids.long().clamp(0, vocab - 1)] + pos.double() + typ.double()[0]
    ref = torch.nn.functional.layer_norm(x, (hidden,), g.double(), b.double(), 1e-12).view(batch * seq, hidden)
    # bf16 rounding of the result, and the fp32 sums of a row
    assert ((buf[: batch * seq].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all()
    assert (buf[batch * seq] == 7.0).all()

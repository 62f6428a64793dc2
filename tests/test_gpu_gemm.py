"""Numerics of the tcgen05 GEMM and implicit-GEMM convolution against plain PyTorch fp32."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch

    assert torch.cuda.is_available()
    torch.cuda.set_device(0)
    torch.manual_seed(0)
    from splitrpc_b200 import ops

    return torch, ops


def _rel_err(torch, got, ref):
    return ((got.float() - ref).norm() / ref.norm().clamp_min(1e-6)).item()


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 128, 512), (256, 384, 1024), (8192, 768, 768),
                                   (100, 200, 72), (4096, 3072, 768), (64, 10, 2048), (3136, 64, 64)])
def test_gemm_plain(env, M, N, K):
    torch, ops = env
    a = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.5).bfloat16()
    out = ops.gemm(a, b)
    ops.check_status()
    ref = a.float() @ b.float().t()
    assert _rel_err(torch, out, ref) < 1e-2


@pytest.mark.parametrize("act", [None, "relu", "gelu"])
def test_gemm_epilogue(env, act):
    torch, ops = env
    M, N, K = 512, 320, 256
    a = (torch.randn(M, K, device="cuda") * 0.3).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.3).bfloat16()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, N, device="cuda").bfloat16()
    out = ops.gemm(a, b, bias=bias, residual=res, act=act)
    ops.check_status()
    ref = a.float() @ b.float().t() + bias + res.float()
    if act == "relu":
        ref = torch.relu(ref)
    elif act == "gelu":
        ref = torch.nn.functional.gelu(ref)
    assert _rel_err(torch, out, ref) < 1e-2
    out32 = ops.gemm(a, b, bias=bias, out_dtype=torch.float32)
    ref32 = a.float() @ b.float().t() + bias
    assert _rel_err(torch, out32, ref32) < 2e-3


@pytest.mark.parametrize("M,N,K", [(4096, 768, 3072), (4096, 1536, 768), (1000, 576, 1024)])
def test_gemm_wide_tiles_with_epilogue(env, M, N, K):
    """Shapes that select the 192-column tile (N a multiple of 192); long K keeps the residual on plain loads."""
    torch, ops = env
    a = (torch.randn(M, K, device="cuda") * 0.2).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.2).bfloat16()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, N, device="cuda").bfloat16()
    out = ops.gemm(a, b, bias=bias, residual=res, act="gelu")
    ops.check_status()
    ref = torch.nn.functional.gelu(a.float() @ b.float().t() + bias + res.float())
    assert _rel_err(torch, out, ref) < 1e-2


@pytest.mark.parametrize("M,N,K", [(4352, 1536, 512), (4097, 1032, 768), (3000, 1000, 832), (2600, 768, 1096), (2049, 128, 2048)])
@pytest.mark.parametrize("ldr_extra", [0, 1, 6])
def test_gemm_pair_tiles_ragged(env, M, N, K, ldr_extra):
    """Edges of the CTA-pair tiles: last rows and columns, K remainders, one to three tiles per pair, residual rows of any stride."""
    torch, ops = env
    a = (torch.randn(M, K, device="cuda") * 0.3).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.3).bfloat16()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, N + ldr_extra, device="cuda").bfloat16()[:, :N]
    buf = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    for act in (None, "relu", "gelu"):
        out = ops.gemm(a, b, bias=bias, residual=res, act=act, out=buf[:M, :N])
        ops.check_status()
        ref = a.double() @ b.double().t() + bias.double() + res.double()
        ref = torch.relu(ref) if act == "relu" else (torch.nn.functional.gelu(ref) if act == "gelu" else ref)
        # half a unit of bf16 (2^-9 of the value) twice, and the fp32 sums: K 2^-24 times the sum of |products| (about 0.09 K)
        assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + K * K * 0.09 * 2.0 ** -24 + 1e-6).all()
        assert (buf[M] == 7.0).all() and (buf[:, N:] == 7.0).all()



def test_gelu_epilogue_matches_erf_definition(env):
    """The epilogue's rational erfc approximation against torch's exact GELU over a wide range of inputs."""
    torch, ops = env
    x = torch.linspace(-8, 8, 128 * 256, device="cuda").view(128, 256)
    eye = torch.eye(256, device="cuda").bfloat16()
    out = ops.gemm(x.bfloat16(), eye, act="gelu", out_dtype=torch.float32)
    ops.check_status()
    ref = torch.nn.functional.gelu(x.bfloat16().float())
    assert (out - ref).abs().max().item() < 2e-6


def test_gelu_epilogue_at_the_ends(env):
    """Infinities, NaN, large and tiny arguments through every kernel that has the epilogue: fp32 by the one-SM kernel, bf16 by CTA
    pairs, both by the first-generation kernel."""
    import math
    torch, ops = env
    x = [math.inf, -math.inf, math.nan, 3e38, -3e38, 70.0, -70.0, 14.0, -14.0, 0.0, -0.0, 1e-30, -1e-30, 1e-40, -1e-40, 5.5, -5.5, 1.0, -1.0]
    bias = torch.tensor(x + [0.5] * (64 - len(x)), device="cuda")
    a, b = torch.zeros(3, 64, device="cuda").bfloat16(), torch.zeros(64, 64, device="cuda").bfloat16()
    ref = torch.nn.functional.gelu(bias.double())
    ref[1] = 0.0  # the limit; the product of infinity and zero is not a number there
    for impl in (1, 2):
        for dtype in (torch.float32, torch.bfloat16):
            ops.GEMM_IMPL, keep = impl, ops.GEMM_IMPL
            try:
                out = ops.gemm(a, b, bias=bias, act="gelu", out_dtype=dtype)
            finally:
                ops.GEMM_IMPL = keep
            ops.check_status()
            out, want = out.double(), ref.expand(3, 64)
            assert torch.equal(out.isnan(), want.isnan())
            assert torch.equal(out[want.isinf()], want[want.isinf()])
            # 7.1.26's 1.5e-7 times |x| / 2 and fp32 rounding; bf16 rounds once more
            tol = 2e-7 * bias.double().abs().clamp(max=6.0) + want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22) + 1e-37
            fin = want.isfinite()
            assert ((out - want).abs() <= tol)[fin].all(), (impl, dtype)
    ops.check_status()


@pytest.mark.parametrize("n,oh,c1,h2,c2,cout,stride2", [(2, 56, 64, 56, 64, 256, 1), (3, 28, 128, 56, 256, 512, 2),
                                                        (2, 14, 256, 28, 512, 1024, 2), (5, 7, 512, 14, 1024, 2048, 2)])
def test_two_input_pointwise_conv(env, n, oh, c1, h2, c2, cout, stride2):
    """Last bottleneck convolution + projection shortcut as one kernel vs the two convolutions in fp32."""
    torch, ops = env
    x1 = (torch.randn(n, oh, oh, c1, device="cuda") * 0.5).bfloat16()
    x2 = (torch.randn(n, h2, h2, c2, device="cuda") * 0.5).bfloat16()
    w1 = (torch.randn(cout, c1, device="cuda") * 0.1).bfloat16()
    w2 = (torch.randn(cout, c2, device="cuda") * 0.1).bfloat16()
    bias = torch.randn(cout, device="cuda")
    out = ops.conv1x1_dual(x1, x2, torch.cat([w1, w2], dim=1).contiguous(), bias=bias, stride2=stride2, act="relu")
    ops.check_status()
    ref = x1.float() @ w1.float().t() + x2[:, ::stride2, ::stride2].float() @ w2.float().t() + bias
    assert out.shape == ref.shape
    assert _rel_err(torch, out, torch.relu(ref)) < 1e-2


@pytest.mark.parametrize("narrow,second", [(64, False), (128, False), (64, True)])
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (1, 8, 16), (2, 13, 11), (7, 56, 56), (40, 31, 31)])
def test_expansion_and_reduction_in_one_kernel(env, n, h, w, narrow, second):
    """One pixel, one whole tile, a ragged last tile, more tiles than SMs: the bits of the two separate kernels, nothing behind them."""
    torch, ops = env
    px, k = n * h * w, 128 if second else 64
    x, x2 = ((torch.randn(n, h, w, 64, device="cuda")).bfloat16() for _ in range(2))
    residual = torch.randn(n, h, w, 256, device="cuda").bfloat16()
    w3, w1 = (torch.randn(256, k, device="cuda") * 0.1).bfloat16(), (torch.randn(narrow, 256, device="cuda") * 0.1).bfloat16()
    b3, b1 = torch.randn(256, device="cuda"), torch.randn(narrow, device="cuda")
    wide, nar = (torch.full((px + 128, c), 7.0, device="cuda", dtype=torch.bfloat16) for c in (256, narrow))
    ops.conv1x1_chain(x, w3, b3, w1, b1, wide[:px].view(n, h, w, 256), nar[:px].view(n, h, w, narrow),
                      residual=None if second else residual, x2=x2 if second else None)
    ops.check_status()
    a = torch.cat([x, x2], dim=3).view(px, 128) if second else x.view(px, 64)
    want = ops.gemm(a, w3, bias=b3, residual=None if second else residual.view(px, 256), act="relu")
    assert torch.equal(wide[:px], want) and torch.equal(nar[:px], ops.gemm(want, w1, bias=b1, act="relu"))
    assert (wide[px:] == 7.0).all() and (nar[px:] == 7.0).all()
    ref = torch.relu(a.double() @ w3.double().t() + b3 + (0 if second else residual.view(px, 256).double()))
    # half a unit of bf16 (2^-9 of the value), and the fp32 sums: K 2^-24 times the sum of |products| (about 0.064 K)
    assert ((want.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + k * k * 0.064 * 2.0 ** -24 + 1e-6).all()


def _one_sm_conv(torch, ops, x, w, bias=None, residual=None, stride=1, pad=0, act=None, x2=None, stride2=1):
    """The convolution by the one-SM kernel: inputs with strides of their own (here the dense ones) always take it."""
    from splitrpc_b200 import _C

    (n, h, wd, c), (cout, r, s, _) = x.shape, w.shape
    out = torch.empty(n, (h + 2 * pad - r) // stride + 1, (wd + 2 * pad - s) // stride + 1, cout, device="cuda", dtype=torch.bfloat16)
    _C.conv_bf16(x.data_ptr(), w.data_ptr(), n, h, wd, c, cout, r, s, stride, pad, out.data_ptr(), 0 if bias is None else bias.data_ptr(),
                 0 if residual is None else residual.data_ptr(), ops.ACT[act], ops.status_word().data_ptr(),
                 torch.cuda.current_stream().cuda_stream, 2, c, wd * c, h * wd * c,
                 **({} if x2 is None else dict(in2=x2.data_ptr(), h2=x2.shape[1], w2=x2.shape[2], cin2=x2.shape[3], stride2=stride2)))
    return out


@pytest.mark.parametrize("n,h,w,cout,r,s", [(1, 20, 16, 128, 4, 1), (1, 11, 14, 72, 4, 1), (1, 20, 16, 128, 2, 1), (1, 20, 16, 200, 3, 1), (2, 20, 16, 64, 4, 1)])
def test_conv_with_few_wide_load_groups(env, n, h, w, cout, r, s):
    """Short filters on small images in the one-SM kernel: all row taps of a column travel in one load group, and the ring holds one to
    three.  CTA pairs, which dense inputs take, give the same bits."""
    torch, ops = env
    x = torch.randn(n, h, w, 64, device="cuda").bfloat16()
    f = (torch.randn(cout, r, s, 64, device="cuda") / (64 * r * s) ** 0.5).bfloat16()
    out = _one_sm_conv(torch, ops, x, f)
    ops.check_status()
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), f.double().permute(0, 3, 1, 2)).permute(0, 2, 3, 1)
    assert out.shape == ref.shape and ((out.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8  # one rounding to bf16
    assert torch.equal(ops.conv2d_nhwc(x, f), out)


@pytest.mark.parametrize("n,oh,c1,h2,c2,cout,stride2", [(2, 14, 64, 14, 64, 256, 1), (3, 9, 128, 17, 64, 72, 2), (2, 7, 512, 14, 256, 512, 2), (1, 30, 64, 90, 64, 64, 3)])
def test_two_inputs_in_the_one_sm_kernel(env, n, oh, c1, h2, c2, cout, stride2):
    """The two-input form for inputs with strides of their own gives the bits of CTA pairs."""
    torch, ops = env
    x1, x2 = torch.randn(n, oh, oh, c1, device="cuda").bfloat16(), torch.randn(n, h2, h2, c2, device="cuda").bfloat16()
    w = (torch.randn(cout, c1 + c2, device="cuda") / (c1 + c2) ** 0.5).bfloat16()
    bias = torch.randn(cout, device="cuda")
    out = _one_sm_conv(torch, ops, x1, w.view(cout, 1, 1, c1 + c2), bias, act="relu", x2=x2, stride2=stride2)
    got = ops.conv1x1_dual(x1, x2, w, bias=bias, stride2=stride2, act="relu")
    ops.check_status()
    ref = torch.relu(x1.double() @ w[:, :c1].double().t() + x2[:, ::stride2, ::stride2].double() @ w[:, c1:].double().t() + bias.double())
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8  # one rounding to bf16
    assert torch.equal(got, out)


@pytest.mark.parametrize("n,h,cin,cout,r,stride,pad", [(2, 56, 64, 64, 3, 1, 1), (4, 28, 128, 128, 3, 1, 1),
                                                       (2, 56, 256, 128, 1, 2, 0), (3, 14, 256, 256, 3, 1, 1),
                                                       (2, 7, 512, 512, 3, 1, 1), (2, 56, 64, 256, 1, 1, 0),
                                                       (2, 28, 128, 128, 3, 2, 1)])
def test_conv_implicit_gemm(env, n, h, cin, cout, r, stride, pad):
    torch, ops = env
    x = (torch.randn(n, h, h, cin, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(cout, r, r, cin, device="cuda") * 0.1).bfloat16()
    bias = torch.randn(cout, device="cuda")
    out = ops.conv2d_nhwc(x, w, bias=bias, stride=stride, pad=pad, act="relu")
    ops.check_status()
    ref = torch.nn.functional.conv2d(x.float().permute(0, 3, 1, 2), w.float().permute(0, 3, 1, 2), bias, stride, pad)
    ref = torch.relu(ref).permute(0, 2, 3, 1)
    assert out.shape == ref.shape
    assert _rel_err(torch, out, ref) < 1e-2
    res = torch.randn_like(out)
    out2 = ops.conv2d_nhwc(x, w, bias=bias, residual=res, stride=stride, pad=pad, act="relu")
    ref2 = torch.relu(torch.nn.functional.conv2d(x.float().permute(0, 3, 1, 2), w.float().permute(0, 3, 1, 2), bias, stride,
                                                 pad).permute(0, 2, 3, 1) + res.float())
    assert _rel_err(torch, out2, ref2) < 1e-2


@pytest.mark.parametrize("M", [1, 64, 65, 128, 129, 200, 300])
@pytest.mark.parametrize("N,K", [(8, 64), (72, 200), (64, 1096), (136, 72), (1000, 512)])
def test_gemm_few_rows(env, M, N, K):
    """Pair tiles of 64 rows per CTA: rows of one CTA only, column halves, odd numbers of k-blocks, a K remainder."""
    torch, ops = env
    a = (torch.randn(M, K, device="cuda") * 0.3).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.3).bfloat16()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, N, device="cuda").bfloat16()
    buf = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    for r in (None, res):
        out = ops.gemm(a, b, bias=bias, residual=r, act="gelu", out=buf[:M, :N])
        ops.check_status()
        ref = a.double() @ b.double().t() + bias.double()
        ref = torch.nn.functional.gelu(ref if r is None else ref + r.double())
        # bounds as in test_gemm_pair_tiles_ragged
        assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + K * K * 0.09 * 2.0 ** -24 + 1e-6).all()
        assert (buf[M] == 7.0).all() and (buf[:, N:] == 7.0).all()


@pytest.mark.parametrize("N,K,act,residual", [(256, 64, "relu", True), (128, 256, "gelu", True), (256, 512, None, True), (1000, 832, "gelu", False),
                                              (768, 3072, None, True), (64, 1024, "relu", False), (192, 40, None, True)])
def test_gemm_rows_do_not_depend_on_their_number(env, N, K, act, residual):
    """A row's bits through every kernel and tile that the number of rows selects: 128- and 256-row pairs of all widths, the one-SM
    kernel, the residual by TMA on both sides of its lines."""
    torch, ops = env
    rows = [1, 64, 129, 700, 2100, 5000, 9000, 14000, 19000, 29000, 45000, 60000]
    rows = [m for m in rows if m * (N + K) <= 6e7]
    a = torch.randn(rows[-1], K, device="cuda").bfloat16()
    b = (torch.randn(N, K, device="cuda") / K ** 0.5).bfloat16()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(rows[-1], N, device="cuda").bfloat16() if residual else None
    whole = ops.gemm(a, b, bias=bias, residual=res, act=act)
    for m in rows[:-1]:
        assert torch.equal(ops.gemm(a[:m], b, bias=bias, residual=res[:m] if residual else None, act=act), whole[:m]), m
    ops.check_status()
    ref = a[:700].double() @ b.double().t() + bias.double() + (res[:700].double() if residual else 0)
    ref = torch.relu(ref) if act == "relu" else (torch.nn.functional.gelu(ref) if act == "gelu" else ref)
    # half a unit of bf16 (2^-9 of the value), and the fp32 sums: K 2^-24 times the sum of |products| (about 0.64 sqrt(K))
    assert ((whole[:700].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + K ** 1.5 * 0.64 * 2.0 ** -24 + 1e-6).all()


@pytest.mark.parametrize("h,w,cin,cout,r,s,stride,pad", [(14, 14, 64, 128, 3, 3, 1, 1), (19, 23, 64, 136, 2, 5, 1, 2), (19, 23, 128, 72, 5, 2, 2, 3),
                                                         (15, 15, 64, 64, 3, 1, 1, 0), (30, 30, 64, 64, 7, 7, 4, 3), (9, 9, 128, 64, 1, 1, 3, 0),
                                                         (7, 7, 512, 512, 3, 3, 1, 1), (5, 5, 64, 8, 3, 3, 2, 1)])
def test_conv_linear_pixels(env, h, w, cin, cout, r, s, stride, pad):
    """Tiles of consecutive output pixels across rows and images: filters of any form, partial last tiles; an image gives the same
    bits in every batch."""
    torch, ops = env
    x = torch.randn(11, h, w, cin, device="cuda").bfloat16()
    wt = (torch.randn(cout, r, s, cin, device="cuda") * 0.05).bfloat16()
    bias = torch.randn(cout, device="cuda")
    ref = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), wt.permute(0, 3, 1, 2).double(), bias.double(), stride, pad).permute(0, 2, 3, 1)
    res = torch.randn(ref.shape, device="cuda").bfloat16()
    K = r * s * cin
    whole = ops.conv2d_nhwc(x, wt, bias=bias, residual=res, stride=stride, pad=pad, act="relu")
    ops.check_status()
    want = torch.relu(ref + res.double())
    # as above, with products of about 0.04 on average
    assert ((whole.double() - want).abs() <= want.abs() * 2.0 ** -8 + K * K * 0.04 * 2.0 ** -24 + 1e-6).all()
    for n in (1, 2, 5):
        part = ops.conv2d_nhwc(x[:n].contiguous(), wt, bias=bias, residual=res[:n].contiguous(), stride=stride, pad=pad, act="relu")
        assert torch.equal(part, whole[:n])
    ops.check_status()


@pytest.mark.parametrize("n,h,w,cin,cout,r,s,stride,pad", [(3, 56, 56, 64, 64, 3, 3, 1, 1), (5, 14, 14, 256, 136, 3, 3, 1, 1), (2, 8, 14, 128, 64, 2, 5, 1, 0),
                                                           (2, 20, 16, 192, 72, 4, 2, 1, 2), (3, 8, 13, 64, 64, 3, 3, 1, 1), (9, 7, 7, 512, 264, 3, 3, 1, 1),
                                                           (2, 20, 20, 64, 64, 5, 5, 1, 2), (2, 28, 28, 128, 128, 3, 3, 2, 1), (3, 9, 30, 64, 200, 1, 1, 1, 0)])
def test_conv_forms_give_the_same_bits(env, n, h, w, cin, cout, r, s, stride, pad):
    """Both sides of the rule for the order of the filter taps: the pair kernel and the one-SM kernel sum alike, residual included."""
    torch, ops = env
    x = torch.randn(n, h, w, cin, device="cuda").bfloat16()
    f = (torch.randn(cout, r, s, cin, device="cuda") / (cin * r * s) ** 0.5).bfloat16()
    bias = torch.randn(cout, device="cuda")
    want = _one_sm_conv(torch, ops, x, f, bias, None, stride, pad, "relu")
    res = torch.randn_like(want)
    for q in (None, res):
        got = ops.conv2d_nhwc(x, f, bias=bias, residual=q, stride=stride, pad=pad, act="relu")
        assert torch.equal(got, want if q is None else _one_sm_conv(torch, ops, x, f, bias, res, stride, pad, "relu"))
    ops.check_status()
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), f.double().permute(0, 3, 1, 2), bias.double(), stride, pad)
    ref = torch.relu(ref.permute(0, 2, 3, 1))
    assert ((want.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8  # one rounding to bf16

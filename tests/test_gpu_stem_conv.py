"""The convolution over overlapping windows of narrow pixels at small and odd image sizes, against an fp64 convolution."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 4, 1), (2, 5, 3), (3, 7, 20), (1, 40, 112), (5, 115, 112), (2, 300, 60)])
@pytest.mark.parametrize("act,gap", [("relu", 0), (None, 48)])
def test_overlapping_windows(C, n, h, w, act, gap):
    import torch
    from splitrpc_b200 import ops

    torch.cuda.set_device(0)
    torch.manual_seed(h * w)
    pitch, oh = w + 3, h - 3
    img = h * pitch * 16 + gap  # elements from one image to the next
    x = torch.randn(n * img + 64, device="cuda").bfloat16()
    wt = (torch.randn(64, 4, 1, 64, device="cuda") / 16).bfloat16()
    bias = torch.randn(64, device="cuda")
    out = torch.full((n * oh * w * 64 + 64,), 7.0, device="cuda", dtype=torch.bfloat16)
    C.conv_bf16(x.data_ptr(), wt.data_ptr(), n, h, w, 64, 64, 4, 1, 1, 0, out.data_ptr(), bias.data_ptr(), 0, ops.ACT[act],
                ops.status_word().data_ptr(), torch.cuda.current_stream().cuda_stream, 2, 16, pitch * 16, img)
    ops.check_status()
    xi = torch.stack([x[i * img:i * img + h * pitch * 16].view(h, pitch, 16) for i in range(n)]).double().permute(0, 3, 1, 2)
    filt = wt.double().view(64, 4, 4, 16).permute(0, 3, 1, 2)  # [out, channel, row tap, pixel of the window]
    ref = torch.nn.functional.conv2d(xi, filt, bias.double()).permute(0, 2, 3, 1)
    ref = torch.relu(ref) if act else ref
    got = out[:-64].view(n, oh, w, 64).double()
    assert ((got - ref).norm() / ref.norm()).item() < 2.0 ** -8  # one rounding to bf16
    assert (got - ref).abs().max().item() < 2.0 ** -7 * ref.abs().max().item()
    assert bool((out[-64:] == 7).all())


@pytest.mark.parametrize("n,h,w", [(1, 4, 1), (2, 7, 20), (3, 12, 40), (2, 115, 112)])
@pytest.mark.parametrize("cout,act", [(128, "relu"), (72, None), (64, "gelu"), (64, "tanh")])
def test_windows_outside_the_stem_kernel(C, n, h, w, cout, act):
    """Output widths and activations that the stem kernel does not have: the one-SM convolution with its row-tap reuse or, on small
    images, its patches."""
    import torch
    from splitrpc_b200 import ops

    torch.cuda.set_device(0)
    torch.manual_seed(h * w + cout)
    pitch, oh = w + 3, h - 3
    img = h * pitch * 16
    x = torch.randn(n * img + 64, device="cuda").bfloat16()
    wt = (torch.randn(cout, 4, 1, 64, device="cuda") / 16).bfloat16()
    bias = torch.randn(cout, device="cuda")
    out = torch.full((n * oh * w * cout + 64,), 7.0, device="cuda", dtype=torch.bfloat16)
    C.conv_bf16(x.data_ptr(), wt.data_ptr(), n, h, w, 64, cout, 4, 1, 1, 0, out.data_ptr(), bias.data_ptr(), 0, ops.ACT[act],
                ops.status_word().data_ptr(), torch.cuda.current_stream().cuda_stream, 2, 16, pitch * 16, img)
    ops.check_status()
    xi = torch.stack([x[i * img:(i + 1) * img].view(h, pitch, 16) for i in range(n)]).double().permute(0, 3, 1, 2)
    filt = wt.double().view(cout, 4, 4, 16).permute(0, 3, 1, 2)  # [out, channel, row tap, pixel of the window]
    ref = torch.nn.functional.conv2d(xi, filt, bias.double()).permute(0, 2, 3, 1)
    ref = {None: ref, "relu": torch.relu(ref), "gelu": torch.nn.functional.gelu(ref), "tanh": torch.tanh(ref)}[act]
    got = out[:-64].view(n, oh, w, cout).double()
    assert ((got - ref).norm() / ref.norm()).item() < 2.0 ** -8  # one rounding to bf16
    assert bool((out[-64:] == 7).all())

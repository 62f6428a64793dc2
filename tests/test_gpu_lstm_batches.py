"""The LSTM app over batch sizes around its groups of eight, plain launches and graphs, against fp64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, L, T = 256, 8, 8


def _exact(w, x):
    sig = lambda v: 1.0 / (1.0 + np.exp(-v))
    seq = [x[:, t].astype(np.float64) for t in range(T)]
    for l in range(L):
        wi, wh, b = (w[3 * l + k].reshape(4 * H, -1).astype(np.float64) for k in range(3))
        h = c = np.zeros((x.shape[0], H))
        out = []
        for v in seq:
            i, g, f, o = np.split(v @ wi.T + h @ wh.T + b[:, 0], 4, axis=1)
            c = sig(f) * c + sig(i) * np.tanh(g)
            h = np.tanh(c) * sig(o)
            out.append(h)
        seq = out
    return seq[-1]


@pytest.mark.parametrize("launch_type", [1, 4])
def test_batches_and_repeated_runs(C, launch_type):
    import torch

    torch.cuda.set_device(0)
    rng = np.random.default_rng(7)
    w = [(rng.standard_normal(s) * 0.08).astype(np.float32) for _ in range(L) for s in ((4, H, H), (4, H, H), (4, H))]
    C.set_rpc_mtu(8192)
    app = C.make_app("lstm", 0, T * H * 4, H * 4, w, 64, launch_type, 17)
    base = app.req_ring[0]
    for n in (1, 2, 3, 4, 5, 6, 7, 8, 9, 17, 2, 1):  # short batches after long ones must not see their words
        x = rng.standard_normal((n, T, H)).astype(np.float32)
        d = torch.from_numpy(x).cuda()
        C.memcpy_async(base, d.data_ptr(), x.nbytes, 0)
        torch.cuda.synchronize()
        got = torch.zeros(n, H, device="cuda")
        for _ in range(3):
            _, resp = C.local_bench(app, 1, n)
        C.memcpy_async(got.data_ptr(), resp[0], n * H * 4, 0)
        torch.cuda.synchronize()
        want = _exact(w, x)
        # 64 cells of 512-term fp32 sums in a row; measured 2e-7 of the result's norm
        assert np.linalg.norm(got.cpu().numpy() - want) < 2e-6 * np.linalg.norm(want), n


@pytest.mark.parametrize("launch_type", [1, 4])
def test_a_wait_that_runs_out_is_reported(C, monkeypatch, launch_type):
    """With a limit of zero the blocks of the upper layers give up at their first look: the run fails, its rows are NaN, and the
    device serves the next app as before."""
    import torch

    torch.cuda.set_device(0)
    rng = np.random.default_rng(9)
    w = [(rng.standard_normal(s) * 0.08).astype(np.float32) for _ in range(L) for s in ((4, H, H), (4, H, H), (4, H))]
    C.set_rpc_mtu(8192)
    x = rng.standard_normal((3, T, H)).astype(np.float32)
    d = torch.from_numpy(x).cuda()

    def run(app):
        C.memcpy_async(app.req_ring[0], d.data_ptr(), x.nbytes, 0)
        torch.cuda.synchronize()
        _, resp = C.local_bench(app, 1, 3)
        got = torch.zeros(3, H, device="cuda")
        C.memcpy_async(got.data_ptr(), resp[0], 3 * H * 4, 0)
        torch.cuda.synchronize()
        return got.cpu().numpy()

    good = C.make_app("lstm", 0, T * H * 4, H * 4, w, 64, launch_type, 8)
    want = run(good)
    np.testing.assert_allclose(want, _exact(w, x), rtol=1e-4, atol=1e-6)
    monkeypatch.setenv("P2P_RPC_APP_WAIT_MS", "0")
    bad = C.make_app("lstm", 0, T * H * 4, H * 4, w, 64, launch_type, 8)
    monkeypatch.delenv("P2P_RPC_APP_WAIT_MS")
    for _ in range(2):
        with pytest.raises(RuntimeError):
            run(bad)
    got = torch.zeros(3, H, device="cuda")
    C.memcpy_async(got.data_ptr(), bad.resp_ring[0], 3 * H * 4, 0)
    torch.cuda.synchronize()
    assert bool(got.isnan().all())
    np.testing.assert_array_equal(run(good), want)


@pytest.mark.parametrize("server_mode", [1, 2])
def test_a_wait_that_runs_out_counts_as_the_workers(C, monkeypatch, server_mode):
    import torch

    torch.cuda.set_device(0)
    rng = np.random.default_rng(10)
    w = [(rng.standard_normal(s) * 0.08).astype(np.float32) for _ in range(L) for s in ((4, H, H), (4, H, H), (4, H))]
    C.set_rpc_mtu(8192)
    sp, cp = C.make_loopback_pair(8192, 512, "pinned")
    monkeypatch.setenv("P2P_RPC_APP_WAIT_MS", "0")
    app = C.make_app("lstm", 0, T * H * 4, H * 4, w, 64, 1, 1)
    srv = C.Server(sp, req_size=T * H * 4, resp_size=H * 4, server_mode=server_mode, max_batch=1)
    srv.add_replica(app)
    srv.start()
    cli = C.Client(cp, req_size=T * H * 4, resp_size=H * 4, total=8, warmup=0, payload="uniform", n_payloads=1)
    try:
        assert cli.run_closed_loop(1) and cli.received == 8
        assert srv.worker_stats(0)["wait_timeouts"] >= 8
    finally:
        srv.stop()


@pytest.mark.parametrize("n_engines", [1, 2])
def test_beside_resident_copy_engines(C, n_engines):
    """The cooperative launch needs 128 SMs while every resident copy engine (copy type 1) holds blocks on 16 of them.  A launch
    that did not fit would wait until an engine leaves at its idle limit of 200 ms."""
    import torch

    torch.cuda.set_device(0)
    rng = np.random.default_rng(8)
    w = [(rng.standard_normal(s) * 0.08).astype(np.float32) for _ in range(L) for s in ((4, H, H), (4, H, H), (4, H))]
    C.set_rpc_mtu(8192)
    sp, cp = C.make_loopback_pair(8192, 512, "pinned")
    apps = [C.make_app("lstm", 0, T * H * 4, H * 4, w, 64, 1, 8, copy_type=1) for _ in range(n_engines)]
    srv = C.Server(sp, req_size=T * H * 4, resp_size=H * 4, server_mode=2, max_batch=8)
    for app in apps:
        srv.add_replica(app)
    srv.start()
    cli = C.Client(cp, req_size=T * H * 4, resp_size=H * 4, total=192, warmup=32, payload="uniform", verify=True, n_payloads=4)
    try:
        assert cli.run_closed_loop(8) and cli.received == 192
        stats = [srv.worker_stats(k) for k in range(n_engines)]
        assert all(s["wait_timeouts"] == 0 and s["num_batches"] > 0 for s in stats)
        assert cli.post_process()["p99_sojournTime_us"] < 50e3
    finally:
        srv.stop()
    for k in range(4):
        x = np.frombuffer(cli.payload(k), dtype=np.float32).reshape(1, T, H)
        got = np.frombuffer(cli.response(k), dtype=np.float32)
        np.testing.assert_allclose(got, _exact(w, x)[0], rtol=1e-4, atol=1e-6)

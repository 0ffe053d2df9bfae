"""Learned warm start on the GPU: the BF16 tensor-core MLP kernels against the CPU
oracle (forward, the gradient of the mean squared error, Adam), the feature kernel
against its numpy restatement, training, and what the trained network gains over the
plain initial pressure on held-out dam-break geometries.

Tolerances: the oracle rounds to BF16 at the same points as the kernels, and the
remaining differences are FP32 against FP64 accumulation order.  A rounding boundary
can flip for a few activations, so the comparisons are relative to each block's scale:
1e-2 for forward outputs and gradients, 1e-5 for the Adam update and 1e-4 for its
second moment (elementwise FP32; the GPU contracts b2 m + (1 - b2) g^2 into an FMA)."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import mlp as omlp
from oracle import oracle
from tests.cases import assert_close, make_params, make_particles
from warpsph_b200 import _capi, core, learned, ops
from warpsph_b200.core import AdjacencyList

pytestmark = pytest.mark.gpu
BLOCKS = [("W1", 0, 512), ("b1", 512, 576), ("W2", 576, 4672), ("b2", 4672, 4736), ("W3", 4736, 8832), ("b3", 8832, 8896),
          ("w4", 8896, 8960), ("b4", 8960, 8961)]


def random_net(seed):
    rng = np.random.default_rng(seed)
    th = omlp.init_params(seed)
    th[512:576] = 0.1 * rng.standard_normal(64)       # nonzero biases so every path is exercised
    th[4672:4736] = 0.1 * rng.standard_normal(64)
    th[8832:8896] = 0.1 * rng.standard_normal(64)
    th[8960] = 0.2
    return th.astype(np.float32)


@pytest.mark.parametrize("tensor_cores", ["tcgen05", "mma"])
@pytest.mark.parametrize("n", [1, 37, 128, 129, 1000, 20000, 200003])
def test_mlp_forward_matches_oracle(cuda, n, tensor_cores):
    """Both forward kernels against the oracle; 200003 samples give the tcgen05 kernel
    several 128-sample tiles per CTA and a ragged last tile."""
    rng = np.random.default_rng(n)
    th = random_net(1)
    x = rng.standard_normal((n, 8)).astype(np.float32)
    ref, _ = omlp.forward(th, x)
    st = ops.mlp_status(cuda)
    st.zero_()
    out = ops.mlp_forward(torch.from_numpy(th).to(cuda), torch.from_numpy(x).to(cuda), tensor_cores=tensor_cores)
    assert int(st.item()) == 0
    assert_close(out.cpu().numpy(), ref, 1e-2, 1e-2, f"MLP forward ({tensor_cores}) vs oracle")
    assert np.median(np.abs(out.cpu().numpy() - ref)) <= 1e-3 * np.abs(ref).max()
    sc = torch.tensor([2.5], device=cuda)
    out2 = ops.mlp_forward(torch.from_numpy(th).to(cuda), torch.from_numpy(x).to(cuda), sc, tensor_cores=tensor_cores)
    assert torch.allclose(out2, 2.5 * out, rtol=1e-6, atol=0)
    assert int(st.item()) == 0


def test_mlp_forward_tcgen05_matches_mma(cuda):
    """The two tensor-core paths round at the same points; they differ only in the FP32
    accumulation order, which can flip a BF16 activation now and then."""
    rng = np.random.default_rng(5)
    th = torch.from_numpy(random_net(3)).to(cuda)
    x = torch.from_numpy(rng.standard_normal((50000, 8)).astype(np.float32)).to(cuda)
    a = ops.mlp_forward(th, x, tensor_cores="tcgen05")
    b = ops.mlp_forward(th, x, tensor_cores="mma")
    d = (a - b).abs()
    scale = b.abs().max()
    assert float(d.max()) <= 1e-2 * float(scale)
    assert float(d.median()) <= 1e-4 * float(scale)


def test_mlp_forward_tc_rejects_misaligned_features(cuda):
    th = torch.from_numpy(random_net(1)).to(cuda)
    buf = torch.zeros(8 * 64 + 2, device=cuda)
    feats = buf[2:].view(64, 8)
    out = torch.empty(64, device=cuda)
    rc = _capi.lib().sph_mlp_forward_tc(th.data_ptr(), 64, feats.data_ptr(), None, out.data_ptr(), None, None)
    assert rc == _capi.SPH_ERR_BAD_ARG
    # the Python wrapper copies such a view to an aligned buffer
    ref = ops.mlp_forward(th, feats.clone())
    assert torch.equal(ops.mlp_forward(th, feats), ref)


@pytest.mark.parametrize("tc", ["tcgen05", "mma"])
@pytest.mark.parametrize("n", [16, 333, 5000, 70000])
def test_mlp_gradient_matches_oracle(cuda, n, tc):
    """The gradient check: every parameter block of the kernel's MSE gradient against the
    oracle's analytic gradient (itself checked against finite differences on the CPU), for
    the tcgen05 kernel (n = 70000 spreads the tiles over every SM, several per CTA) and the
    mma.sync one."""
    rng = np.random.default_rng(10 + n)
    th = random_net(2)
    x = rng.standard_normal((n, 8)).astype(np.float32)
    t = rng.standard_normal(n).astype(np.float32)
    gref, lref = omlp.grad(th, x, t)
    g, loss = ops.mlp_grad(torch.from_numpy(th).to(cuda), torch.from_numpy(x).to(cuda), torch.from_numpy(t).to(cuda),
                           tensor_cores=tc)
    assert int(ops.mlp_status(cuda).item()) == 0
    g = g.cpu().numpy()
    assert abs(float(loss.item()) - lref) <= 1e-2 * lref
    for name, a, b in BLOCKS:
        assert_close(g[a:b], gref[a:b], 2e-2, 2e-2, f"d loss / d {name}")


def test_mlp_adam_matches_oracle(cuda):
    rng = np.random.default_rng(3)
    th = random_net(3)
    m1 = np.zeros_like(th); m2 = np.zeros_like(th)
    T, M1, M2 = (torch.from_numpy(a.copy()).to(cuda) for a in (th, m1, m2))
    for step in range(1, 4):
        g = (1e-2 * rng.standard_normal(th.shape)).astype(np.float32)
        th, m1, m2 = omlp.adam(th, g, m1, m2, step, 1e-3)
        ops.mlp_adam(T, torch.from_numpy(g).to(cuda), M1, M2, step, 1e-3)
    assert_close(T.cpu().numpy(), th, 1e-5, 1e-6, "Adam parameters")
    assert_close(M2.cpu().numpy(), m2, 1e-4, 1e-6, "Adam second moment (FMA-contracted on the GPU)")


@pytest.mark.parametrize("mode", [0, 1])
def test_dfsph_features_match_numpy(cuda, mode):
    """The eight features restated in numpy on the oracle's divergence, alpha and kernel."""
    cfg, sch, p = make_params(2, kernel=core.KernelFunctions.Wendland4)
    P = make_particles(2, 20, seed=7, jitter=0.3, h_spread=0.1)
    rng = np.random.default_rng(8)
    n = len(P["masses"])
    x, H, m, v = P["positions"], P["supports"], P["masses"], P["velocities"]
    dvdt = (0.3 * rng.standard_normal(x.shape)).astype(np.float32)
    pprev = (0.2 + 0.1 * rng.random(n)).astype(np.float32)
    o = oracle.get("f32")
    nb = o.neighbors(p, x, H, 1 << 14)
    rho = o.density(p, 0, x, H, m, nb)
    dt, rho0 = np.float32(2e-3), 1.0
    div = o.incompressible_divergence(p, rho0, x, H, m, rho, v, dvdt, dt, nb)
    al = o.dfsph_alpha(p, x, H, m, rho, nb)
    if mode == 0:
        src, diag = -div, dt * al
    else:
        src = np.float32(rho0) - np.maximum(rho + dt * div, np.float32(0.9))
        diag = np.minimum((dt * dt) * al, np.float32(-1e-6))
    pj = (src / diag).astype(np.float64)
    Pref = np.abs(pj).mean()
    S = np.zeros((n, 3))
    for i in range(n):
        row = nb["list"][nb["offsets"][i]: nb["offsets"][i] + nb["counts"][i]]
        d = x[i] - x[row]
        d = np.where(d > 0.5, d - 1, np.where(d < -0.5, d + 1, d))
        W, _, _ = o.kernel_eval(p.kernel, 2, np.linalg.norm(d, axis=1), float(H[i]))
        w = m[row] / rho[row] * W
        S[i] = [w.sum(), (w * pj[row]).sum(), (w * pprev[row]).sum()]
    cnt = nb["counts"].astype(np.float64)
    ref = np.stack([pj / Pref, S[:, 1] / Pref, pprev / Pref, S[:, 2] / Pref, 100 * (rho / rho0 - 1), S[:, 0] - 1,
                    cnt / cnt.mean() - 1, diag / diag.mean() - 1], 1)
    t = {k: torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for k, a in dict(x=x, H=H, m=m, rho=rho, v=v, dvdt=dvdt, pp=pprev).items()}
    adj = AdjacencyList(neighborOffsets=torch.from_numpy(nb["offsets"]).to(cuda), numNeighbors=torch.from_numpy(nb["counts"]).to(cuda),
                        neighborList=torch.from_numpy(nb["list"]).to(cuda), numRows=n, numCols=n, nnz=int(nb["nnz"]))
    c = _capi.SphJacobiConfig()
    c.rest_density = rho0
    f, sc = ops.dfsph_features(p, mode, c, t["x"], t["H"], t["m"], t["rho"], t["v"], t["dvdt"], t["pp"], float(dt), adj)
    assert abs(float(sc.item()) - Pref) <= 1e-4 * Pref
    for k in range(8):
        assert_close(f.cpu().numpy()[:, k], ref[:, k], 1e-4, 1e-4, f"feature {k}")


def test_training_reduces_loss(cuda):
    """Adam on the kernels' gradient fits a smooth function of the features."""
    rng = np.random.default_rng(4)
    x = rng.standard_normal((20000, 8)).astype(np.float32)
    y = (np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2] - 0.3 * np.abs(x[:, 3])).astype(np.float32)
    X, Y = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
    net = learned.WarmStartMLP(cuda, seed=0)
    l0 = net.loss(X, Y)
    losses = net.fit(X, Y, epochs=25, batch=2048, lr=3e-3)
    assert losses[-1] < 0.1 * l0 and losses[-1] < losses[0]


def test_learned_warm_start_gain(cuda):
    """What the trained network gains: on dam-break column sizes it was not trained on,
    the density solve reaches the 0.01 % tolerance in at most 0.7 of the plain solve's
    iterations, from the same states and to the same stopping rule, with no missed
    tolerance.  (The divergence-free learned start is trained and reported by bench.py
    but shows no gain in a free-surface column: that solve stalls above its tolerance
    there, so its targets are not converged pressures.)"""
    rng = np.random.default_rng(0)
    geos = [(float(rng.uniform(0.3, 0.7)), float(rng.uniform(0.6, 1.0)), s) for s in range(6)]
    data = learned.generate_samples(geos, steps=10, device=cuda, dx=0.02)
    nets = []
    for mode in (1, 0):
        f, tg = data[mode]
        net = learned.WarmStartMLP(cuda, seed=mode)
        losses = net.fit(f, tg, epochs=25, batch=4096, lr=2e-3)
        assert losses[-1] < 0.5 * float(tg.var())
        nets.append(net)
    tot = learned.compare_warm_starts([(0.45, 0.85, 100), (0.62, 0.72, 101)], steps=8, nets=(nets[0], nets[1]), device=cuda, dx=0.02)
    d = tot["density"]
    assert d["learned"][2] == 0 and d["plain"][2] == 0, d
    assert d["learned"][0] <= 0.7 * d["plain"][0], d


@pytest.mark.parametrize("tiles", [1, 147, 148, 149, 2 * 148, 3 * 148 + 1, 4 * 148 - 1, 7 * 148 + 5])
def test_mlp_gradient_adds_up(cuda, tiles):
    """The gradient over 2 m samples against the mean of those over its halves, m = 128 x tiles, for
    every number of tiles per SM modulo the three in flight.  dy of a half is exactly twice that of
    the whole, so all BF16 roundings agree and only the FP32 sums are ordered differently: 2e-4 of
    a block's largest entry is 3000 roundings of it."""
    m = 128 * tiles
    rng = np.random.default_rng(tiles)
    th = torch.from_numpy(random_net(3)).to(cuda)
    x = torch.from_numpy(rng.standard_normal((2 * m, 8)).astype(np.float32)).to(cuda)
    t = torch.from_numpy(rng.standard_normal(2 * m).astype(np.float32)).to(cuda)
    g, loss = ops.mlp_grad(th, x, t, tensor_cores="tcgen05")
    (ga, la), (gb, lb) = (ops.mlp_grad(th, x[s], t[s], tensor_cores="tcgen05") for s in (slice(0, m), slice(m, 2 * m)))
    assert int(ops.mlp_status(cuda).item()) == 0
    ref = 0.5 * (ga.double() + gb.double())
    for name, a, b in BLOCKS:
        assert_close(g[a:b].cpu().numpy(), ref[a:b].cpu().numpy(), 2e-4, 2e-4, f"d loss / d {name}")
    assert abs(float(loss) - (float(la) + float(lb))) <= 1e-6 * float(loss)        # the loss is a sum


@pytest.mark.parametrize("n", [1, 127, 128, 129, 5 * 148 * 128 + 1, 6 * 148 * 128 - 5, 11 * 148 * 128 + 300])
def test_mlp_forward_is_per_row(cuda, n):
    """The tcgen05 forward of n rows against the same rows evaluated in slices: a row's output
    does not depend on the tile, the warpgroup or the SM that computes it, so they are equal."""
    rng = np.random.default_rng(n % 1000)
    th = torch.from_numpy(random_net(4)).to(cuda)
    x = torch.from_numpy(rng.standard_normal((n, 8)).astype(np.float32)).to(cuda)
    y = ops.mlp_forward(th, x)
    step = 1000 if n < 10**5 else 200_000
    ref = torch.cat([ops.mlp_forward(th, x[a:a + step]) for a in range(0, n, step)])
    assert int(ops.mlp_status(cuda).item()) == 0
    assert torch.equal(y, ref)


def test_gradient_reports_an_issuing_warp_that_gave_up(cuda, tmp_path):
    """The kernel compiled with a stand-in for a wait that runs out before a block's last weight-gradient
    product: each of 200 such launches returns the timeout status, and plain launches around them none and the same
    gradient (1e-5 of its largest entry: its FP32 atomics add 148 partial sums in another order)."""
    import subprocess
    from pathlib import Path
    from warpsph_b200 import build
    src = Path(__file__).resolve().parent / "native" / "mlp_give_up_check.cu"
    exe = tmp_path / "mlp_give_up_check"
    subprocess.run([build.nvcc(), *build.ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.INCLUDE), "-I",
                    str(build.CSRC), str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert out[:8] == ["plain", "0", "given_up", "200", "of", "200", "after", "0"] and float(out[9]) < 1e-5, out


def test_inference_reports_a_single_thread_that_gave_up(cuda, tmp_path):
    """One thread's stand-in for a wait that runs out on the last chain of its warpgroup: NaN in its row
    and the timeout status, neither in the launches around it."""
    import subprocess
    from pathlib import Path
    from warpsph_b200 import build
    src = Path(__file__).resolve().parent / "native" / "mlp_forward_give_up_check.cu"
    exe = tmp_path / "mlp_forward_give_up_check"
    subprocess.run([build.nvcc(), *build.ARCH_FLAGS, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.INCLUDE), "-I",
                    str(build.CSRC), str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert out == ["plain", "0", "0", "given_up", str(_capi.STATUS_TIMEOUT), "1", "after", "0", "0"], out

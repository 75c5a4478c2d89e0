"""The learned warm start's tensor-core kernels (B200).

- The tcgen05 BF16 GEMM against a float64 product of the same BF16 inputs
  (FP32 accumulation: agreement to FP32 rounding), with its fused bias,
  tanh and BF16 epilogue, on ragged row counts, several N tiles and K chunks.
- The network's gradients against the numpy restatement (oracle/mlp_ref.py),
  which rounds to BF16 where the GPU does: relative error of each gradient
  tensor below 1e-3 (FP32 summation order, and a BF16 rounding it flips).
- Training on the GPU fits a smooth map, takes the steps of a host
  restatement, and does not depend on work queued on the default stream; the
  loss of uneven, infinite and NaN errors.
- A completion wait that runs out (every wait bounded to no rounds) raises
  the timeout status and stores nothing; the next unbounded GEMM on the same
  device is correct (the drained MMAs left the context usable).
"""

import subprocess

import numpy as np
import pytest

from espice_b200 import mlp
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    assert torch.cuda.is_available(), "a CUDA device is required"
    return torch


# the last: the learned step's inference shape (a 32,768-point chunk through
# a 512-wide hidden layer)
@pytest.mark.parametrize("M,N,K", [(200, 96, 48), (1000, 512, 512), (128, 16, 16), (333, 272, 80),
                                   (32768, 512, 512)])
def test_gemm_matches_float64(M, N, K):
    torch = _torch()
    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(N, generator=g).cuda()
    c = torch.zeros(M, N, device="cuda")
    h = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    mlp.gemm_bf16(a.data_ptr(), K, b.data_ptr(), K, M, N, K, c.data_ptr(), N, d_bias=bias.data_ptr(),
                  d_h=h.data_ptr(), ldh=N, act=1)
    torch.cuda.synchronize()
    ref = a.double().cpu() @ b.double().cpu().T + bias.double().cpu()
    got = c.double().cpu()
    scale = (a.double().abs().cpu() @ b.double().abs().cpu().T).max()
    assert float((got - ref).abs().max()) <= 1e-6 * float(scale) + 1e-6
    # the BF16 tanh copy: the device's tanhf and the host's may differ in the
    # last FP32 bit, which flips a BF16 rounding now and then: one BF16 ulp,
    # on a handful of the elements at most
    th = torch.tanh(c.cpu()).to(torch.bfloat16).float()
    hb = h.cpu().float()
    assert torch.allclose(hb, th, rtol=2.0 ** -7, atol=0.0)
    assert float((hb != th).float().mean()) <= 1e-5


def test_gemm_without_bias_or_copy():
    torch = _torch()
    M, N, K = 130, 32, 32
    a = torch.randn(M, K).to(torch.bfloat16).cuda()
    b = torch.randn(N, K).to(torch.bfloat16).cuda()
    c = torch.zeros(M, N, device="cuda")
    torch.cuda.synchronize()
    mlp.gemm_bf16(a.data_ptr(), K, b.data_ptr(), K, M, N, K, c.data_ptr(), N)
    torch.cuda.synchronize()
    ref = a.double().cpu() @ b.double().cpu().T
    assert float((c.double().cpu() - ref).abs().max()) < 1e-4


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def test_gradients_match_reference():
    torch = _torch()
    rng = np.random.default_rng(3)
    n_in, n_out, rows = 16, 40, 64
    net = mlp.Mlp(n_in, 64, 3, n_out, seed=5)
    in_mu, in_sig = rng.normal(size=n_in).astype(np.float32), rng.uniform(0.5, 2, n_in).astype(np.float32)
    out_mu, out_sig = rng.normal(size=n_out).astype(np.float32), rng.uniform(0.5, 2, n_out).astype(np.float32)
    net.set_scaling(in_mu, in_sig, out_mu, out_sig)
    x = rng.normal(size=(rows, n_in)).astype(np.float32)
    y = rng.normal(size=(rows, n_out)).astype(np.float32)
    dx, dy = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    torch.cuda.synchronize()
    loss, grads = net.gradients(dx.data_ptr(), dy.data_ptr(), rows)
    layers = net.weights()
    loss_ref, grads_ref = mlp_ref.gradients(layers, x, y, in_mu, in_sig, out_mu, out_sig)
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    for (gw, gb), (rw, rb) in zip(grads, grads_ref):
        assert _rel(gw, rw) < 1e-3
        assert _rel(gb, rb) < 1e-3
    net.close()


def test_training_fits_a_smooth_map():
    torch = _torch()
    rng = np.random.default_rng(11)
    n_in, n_out, n = 4, 24, 4096
    A = rng.normal(size=(n_in, n_out))
    x = rng.uniform(-1, 1, size=(n, n_in)).astype(np.float32)
    y = np.sin(x @ A).astype(np.float32)
    net = mlp.Mlp(n_in, 128, 3, n_out, seed=2)
    net.set_scaling(x.mean(0), x.std(0), y.mean(0), y.std(0))
    dx, dy = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    torch.cuda.synchronize()
    loss = net.train(dx.data_ptr(), dy.data_ptr(), n, epochs=60, batch=256, lr=2e-3)
    assert loss[-1] < 0.05 * loss[0]
    out = torch.zeros(n, n_out, device="cuda")
    net.predict(dx.data_ptr(), n, out.data_ptr())
    torch.cuda.synchronize()
    err = np.abs(out.cpu().numpy() - y).mean()
    assert err < 0.1
    net.close()


@pytest.mark.parametrize("errors,want", [
    ([(0, 2064, 1e-6), (1500, 1501, 1.0)], None),         # far above the sum before its chunk
    ([(1024, 2064, 1e-9), (2050, 2064, 1e3)], None),      # a first chunk without error, then a rise
    ([(0, 2064, 1e-18), (2000, 2001, 1e18)], None),       # near the ends of the range
    ([(0, 1, 1e3), (1, 2064, 1e-3)], None),
    ([(0, 2064, 0.25)], None),
    ([], None),
    ([(0, 2064, 0.25), (3, 4, np.inf)], np.inf),
    ([(2063, 2064, np.inf)], np.inf),
    ([(0, 2064, 0.25), (1100, 1101, 1e25)], np.inf),      # its square past FP32
    ([(0, 2064, 0.25), (7, 8, np.inf), (1999, 2000, np.nan)], np.nan),
    ([(0, 2064, 0.25), (5, 6, np.nan)], np.nan),
])
def test_loss_of_uneven_errors(errors, want):
    """The loss against its FP32 terms summed in FP64, where they are finite:
    2,064 roundings to nearest of a sum of one sign, 2^-24 of it each; an
    infinite term gives infinity, a NaN gives NaN."""
    torch = _torch()
    rows, n_out = 16, 129
    net = mlp.Mlp(4, 16, 2, n_out, seed=9)
    x = torch.linspace(-1.0, 1.0, rows * 4, device="cuda").reshape(rows, 4).contiguous()
    y = torch.zeros(rows, n_out, device="cuda")
    torch.cuda.synchronize()
    net.predict(x.data_ptr(), rows, y.data_ptr())
    t = y.cpu().numpy().ravel().copy()
    out = t.copy()
    for lo, hi, e in errors:
        t[lo:hi] += np.float32(e)
    dt = torch.tensor(t, device="cuda")
    torch.cuda.synchronize()
    loss, _ = net.gradients(x.data_ptr(), dt.data_ptr(), rows)
    net.close()
    with np.errstate(over="ignore", invalid="ignore"):
        e = out - t
        terms = e * e / np.float32(rows * n_out)
    if want is None:
        ref = float(np.sum(terms.astype(np.float64)))
        assert abs(loss - ref) <= rows * n_out * 2.0 ** -24 * ref
    else:
        assert np.array_equal(np.float32(loss), np.float32(want), equal_nan=True)


@pytest.mark.parametrize("passes", [4, 12, 24, 48])
def test_training_beside_work_on_the_default_stream(passes):
    """A run's new buffers are made ready on the network's own stream: work
    queued on the default stream (about a third of a millisecond a pass; it
    ends before, within and after the 64 steps) changes no weight."""
    torch = _torch()
    big = torch.ones(1 << 28, device="cuda")
    g = torch.Generator().manual_seed(2)
    x = torch.randn(16384, 16, generator=g).cuda()
    y = torch.randn(16384, 64, generator=g).cuda()

    def run(queued):
        net = mlp.Mlp(16, 64, 3, 64, seed=3)
        torch.cuda.synchronize()
        for _ in range(queued):
            big.mul_(1.0)
        loss = net.train(x.data_ptr(), y.data_ptr(), len(x), epochs=1, batch=256, lr=1e-3)
        torch.cuda.synchronize()
        weights = np.concatenate([a.ravel() for layer in net.weights() for a in layer])
        net.close()
        return loss, weights

    (la, wa), (lb, wb) = run(passes), run(0)
    assert np.array_equal(la, lb) and np.array_equal(wa.view(np.uint32), wb.view(np.uint32))


SHUFFLE = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
int main(int, char** v) {
  std::mt19937_64 rng(std::strtoull(v[1], nullptr, 10));
  std::vector<unsigned> p(std::atoi(v[2]));
  for (unsigned i = 0; i < p.size(); ++i) p[i] = i;
  for (int e = std::atoi(v[3]); e--;) {
    std::shuffle(p.begin(), p.end(), rng);
    for (unsigned i : p) std::printf("%u ", i);
  }
}
"""


@pytest.fixture(scope="module")
def orders(tmp_path_factory):
    """The runs' sample orders: the C++ library's shuffle of 0 .. n - 1, epoch after epoch."""
    d = tmp_path_factory.mktemp("shuffle")
    (d / "s.cpp").write_text(SHUFFLE)
    subprocess.run(["g++", "-O1", str(d / "s.cpp"), "-o", str(d / "s")], check=True)
    return lambda seed, n, epochs: np.array(
        subprocess.run([str(d / "s"), str(seed), str(n), str(epochs)], check=True, capture_output=True,
                       text=True).stdout.split(), np.int64).reshape(epochs, n)


def test_training_steps_match_the_restatement(orders):
    """Two runs of several epochs and batches of distinct rows on one network,
    the rate decaying: batches, rates and bias corrections as a host
    restatement takes them (the numpy gradients, Adam in FP64). Each step's
    gradients agree to 1e-3 of their norm; of the elements, about that part
    lies below the error and may turn the sign of its step, sqrt(1e-3) = 3%
    of a step's norm, and ten steps add up. A wrong batch, rate or
    correction moves the weights elsewhere altogether."""
    torch = _torch()
    rng = np.random.default_rng(21)
    n_in, n_out, batch, n = 6, 20, 32, 70  # two batches and a rest an epoch
    x = rng.normal(size=(n, n_in)).astype(np.float32)
    y = (np.sin(2.0 * x @ rng.normal(size=(n_in, n_out))) + rng.normal(size=(n, n_out))).astype(np.float32)
    dx, dy = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    torch.cuda.synchronize()
    net = mlp.Mlp(n_in, 48, 3, n_out, seed=6)
    layers = [(w.astype(np.float64), b.astype(np.float64)) for w, b in net.weights()]
    start = np.concatenate([a.ravel() for layer in layers for a in layer])
    mom = [[np.zeros_like(a) for a in layer] for layer in layers]
    var = [[np.zeros_like(a) for a in layer] for layer in layers]
    one = np.ones(max(n_in, n_out), np.float32)
    t = 0
    for epochs, lr, lr_end, seed in ((3, 2e-2, 5e-3, 4), (2, 1e-2, 2e-3, 9)):
        got = net.train(dx.data_ptr(), dy.data_ptr(), n, epochs=epochs, batch=batch, lr=lr, lr_end=lr_end, seed=seed)
        perm = orders(seed, n, epochs)
        for ep in range(epochs):
            rate = lr * (lr_end / lr) ** (ep / (epochs - 1))
            losses = []
            for b in range(n // batch):
                rows = perm[ep][b * batch:(b + 1) * batch]
                loss, grads = mlp_ref.gradients([(w.astype(np.float32), c.astype(np.float32)) for w, c in layers],
                                                x[rows], y[rows], 0 * one[:n_in], one[:n_in], 0 * one[:n_out],
                                                one[:n_out])
                losses.append(loss)
                t += 1
                new = []
                for k, layer in enumerate(layers):
                    out = []
                    for j, a in enumerate(layer):
                        g = grads[k][j].astype(np.float64)
                        mom[k][j] = 0.9 * mom[k][j] + 0.1 * g
                        var[k][j] = 0.999 * var[k][j] + 0.001 * g * g
                        out.append(a - rate * (mom[k][j] / (1 - 0.9 ** t)) / (np.sqrt(var[k][j] / (1 - 0.999 ** t))
                                                                             + 1e-8))
                    new.append(tuple(out))
                layers = new
            assert abs(got[ep] - np.mean(losses)) <= 1e-2 * np.mean(losses)
        want = np.concatenate([a.ravel() for layer in layers for a in layer]) - start
        moved = np.concatenate([a.ravel() for layer in net.weights() for a in layer]) - start
        assert np.linalg.norm(moved - want) <= 0.1 * np.linalg.norm(want)
    net.close()


def test_gemm_wait_runs_out_and_stores_nothing():
    torch = _torch()
    M, N, K = 256, 128, 192
    g = torch.Generator().manual_seed(7)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    c = torch.full((M, N), 12345.0, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(mlp.MlpError) as err:
        mlp.gemm_bf16(a.data_ptr(), K, b.data_ptr(), K, M, N, K, c.data_ptr(), N, wait_rounds=mlp.GEMM_NO_WAIT)
    assert err.value.code == mlp.MLP_TIMEOUT
    torch.cuda.synchronize()
    assert bool((c == 12345.0).all()), "a timed-out GEMM stored results"
    mlp.gemm_bf16(a.data_ptr(), K, b.data_ptr(), K, M, N, K, c.data_ptr(), N)
    torch.cuda.synchronize()
    ref = a.double().cpu() @ b.double().cpu().T
    assert torch.allclose(c.double().cpu(), ref, rtol=1e-5, atol=1e-4)

"""The training step's kernels at other shapes than the benchmark's: batches of one row tile and of
odd numbers of tiles, both hidden widths, K loops shorter and longer than the stages in flight,
features at an address that only allows two-byte loads, and parameters through set and get."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from protlocus_b200 import lib as L

pytestmark = pytest.mark.gpu


def _bf(x):
    return x.to(torch.bfloat16)


@pytest.mark.parametrize("M,N,K,tile", [(128, 64, 64 * k, t) for k in (1, 2, 3, 5, 6, 7, 9, 17) for t in (16, 48, 64)] +
                         [(256, 256, 64 * k, 256) for k in (1, 2, 3, 4, 5, 9)] + [(384, 208, 448, 80)])
def test_gemm_stage_counts(M, N, K, tile):
    g = torch.Generator(device="cpu").manual_seed(M + N + K + tile)
    A = _bf(torch.randn(M, K, generator=g)).cuda()
    B = _bf(torch.randn(N, K, generator=g)).cuda()
    C = torch.zeros(M, N, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert L.load().pl_pf_gemm(0, A.data_ptr(), K, B.data_ptr(), K, M, N, K, tile, None, 0, None, N, None, N, None, M,
                               C.data_ptr(), N, err.data_ptr(), None), L.error()
    torch.cuda.synchronize()
    want = A.double() @ B.double().T
    # fp32 accumulation of K products of magnitude about 1: 2^-24 per addition, K additions at worst
    assert int(err.item()) == 0 and (C.double() - want).abs().max().item() <= K * 2.0 ** -24 * 4 * K ** 0.5


@pytest.mark.parametrize("batch,hidden,shift", [(128, 256, 0), (384, 128, 0), (640, 256, 1), (1152, 128, 1)])
def test_step_against_torch(batch, hidden, shift):
    """One step's parameter change against the gradients of the same loss in torch on the same
    bf16 weights: where the gradient is well away from zero Adam's first step has its sign and is
    lr long (and 1e-5 * lr * w of decay)."""
    lib = L.load()
    g = torch.Generator(device="cpu").manual_seed(batch + hidden)
    rows = 2 * batch
    X = _bf(torch.randn(rows, 576, generator=g).abs() * 0.3)
    y = (torch.rand(rows, generator=g) < 0.4).float()
    s = torch.sort(torch.rand(rows, 2, generator=g), dim=1).values
    T = torch.stack([y, s[:, 0], s[:, 1], y], dim=1)
    perm = torch.randperm(rows, generator=g).to(torch.int32)
    buf = torch.zeros(rows * 576 + 8, dtype=torch.bfloat16, device="cuda")
    buf[shift:shift + rows * 576] = X.reshape(-1).cuda()
    dT, dP = T.cuda(), perm.cuda()
    h = lib.pl_pf_model_create(0, 576, hidden, 5)
    assert h, L.error()
    try:
        n = lib.pl_pf_model_size(h)
        p0, p1 = np.zeros(n, np.float32), np.zeros(n, np.float32)
        assert lib.pl_pf_model_get(h, p0.ctypes.data, n)
        p0 += 0.01 * np.random.default_rng(1).standard_normal(n).astype(np.float32)
        assert lib.pl_pf_model_set(h, p0.ctypes.data, n) and lib.pl_pf_model_get(h, p1.ctypes.data, n)
        assert np.array_equal(p0, p1)
        loss = np.zeros(1, np.float32)
        torch.cuda.synchronize()
        assert lib.pl_pf_train(h, buf.data_ptr() + 2 * shift, dT.data_ptr(), dP.data_ptr(), rows, batch, 1, 1e-3, 4.0, 2.0,
                               loss.ctypes.data, None), L.error()
        assert lib.pl_pf_model_get(h, p1.ctypes.data, n)
    finally:
        lib.pl_pf_model_destroy(h)
    ws, off = [], 0
    for o, i in ((hidden, 576), (hidden, hidden), (hidden, hidden), (16, hidden)):
        W = torch.from_numpy(p0[off:off + o * i].copy()).reshape(o, i)
        b = torch.from_numpy(p0[off + o * i:off + o * i + o].copy())
        ws.append((_bf(W).double().requires_grad_(), b.double().requires_grad_()))
        off += o * i + o
    rows_ = perm[:batch].long()
    a, t = X[rows_].double(), T[rows_].double()
    for k, (W, b) in enumerate(ws):
        a = a @ W.T + b
        if k < 3:
            a = torch.relu(a)
            a = a + (_bf(a).double() - a).detach()  # activations rounded as on the device
    cw = torch.where(t[:, 0] > 0.5, 4.0, 1.0)
    bce = torch.nn.functional.binary_cross_entropy_with_logits(a[:, 0], t[:, 0], reduction="none")
    d = (a[:, 1:3] - t[:, 1:3]).abs()
    tot = (cw * bce + 2.0 * t[:, 3] * torch.where(d < 0.05, d * d / 0.1, d - 0.025).sum(1)).mean()
    assert abs(tot.item() - float(loss[0])) <= 2e-2 * abs(tot.item())  # bf16 activations
    tot.backward()
    gr = torch.cat([x.grad.reshape(-1) for W, b in ws for x in (W, b)]).numpy()
    step = (p1 - p0).astype(np.float64)
    big = np.abs(gr) > 0.05 * np.abs(gr).max()
    assert big.sum() > 100
    assert (np.sign(step[big]) == -np.sign(gr[big])).mean() > 0.98
    right = big & (np.sign(step) == -np.sign(gr))
    assert np.allclose(np.abs(step[right]), 1e-3, rtol=1e-3, atol=1e-3 * 1e-5 * 2)

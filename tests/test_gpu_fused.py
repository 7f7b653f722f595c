"""The two-launch schedule of small matrices (HM_OPT_OVERLAP 2, the default)
against the stage-by-stage schedules: the same sums in the same order, so equal
bit for bit.  Sizes from one leaf to beyond the last size that takes it, ranks
with and without unrolled kernels, strided and accumulating calls, the
transposed and derivative products, and a replayed CUDA graph."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

TDT = {"f64": torch.float64, "f32": torch.float32, "df64": torch.float64}
STORE = {"f64": np.float64, "f32": np.float32, "df64": "df64"}


def matrix(n, m, dtype, rank=20, kernel=hm.cauchykernel):
    rng = np.random.default_rng(n + m)
    x, y = np.sort(rng.random(n))[::-1].copy(), np.sort(rng.random(m))[::-1].copy()
    return hm.KernelMatrix(kernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=STORE[dtype], rank=rank)


def vectors(rows, k, dtype, seed):
    v = torch.randn(k, rows, device="cuda", dtype=TDT[dtype], generator=torch.Generator("cuda").manual_seed(seed)).t()
    return v[:, 0].contiguous() if k == 1 else v


@pytest.mark.parametrize("dtype", ["f64", "f32", "df64"])
@pytest.mark.parametrize("n,m,rank", [(40, 40, 20), (200, 170, 20), (1000, 1000, 20), (2049, 1777, 13), (5000, 4000, 20),
                                      (9001, 9001, 20)])
@pytest.mark.parametrize("k", [1, 2, 3, 8, 9, 17])
def test_equals_stage_schedules(dtype, n, m, rank, k):
    H = matrix(n, m, dtype, rank)
    X, U0 = vectors(m, k, dtype, 1), vectors(n, k, dtype, 2)
    for acc in (False, True):
        U = U0.clone()
        H.mul(U, X, accumulate=acc)
        H.set_overlap(1)
        V = U0.clone()
        H.mul(V, X, accumulate=acc)
        H.set_overlap(True)
        assert torch.equal(U, V)
    assert H.device_status() == 0
    H.free()


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_strided_transposed_and_derivative_products(dtype):
    H = matrix(1500, 1200, dtype)
    x = vectors(1 + 2 * 1200, 1, dtype, 3)
    got, ref = torch.zeros(5 + 3 * 1500, device="cuda", dtype=TDT[dtype]), torch.zeros(5 + 3 * 1500, device="cuda", dtype=TDT[dtype])
    w, g = vectors(1200, 1, dtype, 4), vectors(1500, 1, dtype, 5)
    H.mul_strided(got, x, 5, 2, 2, 3)
    fused = [got, H.T @ g, H.mul_drow(torch.empty_like(g), w, accumulate=False),
             H.mul_drow(torch.empty_like(w), g, transposed=True, accumulate=False)]
    H.set_overlap(1)
    H.mul_strided(ref, x, 5, 2, 2, 3)
    staged = [ref, None, H.mul_drow(torch.empty_like(g), w, accumulate=False), None]
    for a, b in zip(fused, staged):
        assert b is None or torch.equal(a, b)
    D = 1.0 / (torch.tensor(H.x)[:, None] - torch.tensor(H.y)[None, :])
    tol = 1e-12 if dtype == "f64" else 1e-6
    rt = D.t() @ g.double().cpu()
    assert float(torch.linalg.norm(fused[1].double().cpu() - rt) / torch.linalg.norm(rt)) <= tol
    rd = (D * D).t() @ g.double().cpu()
    assert float(torch.linalg.norm(fused[3].double().cpu() - rd) / torch.linalg.norm(rd)) <= max(tol, 1e-11)
    H.free()


@pytest.mark.parametrize("dtype", ["f64", "f32", "df64"])
def test_graph_replay_and_streams(dtype):
    H = matrix(3000, 2500, dtype)
    x = vectors(2500, 1, dtype, 6)
    ref = H @ x
    u, s = torch.empty_like(ref), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        H.mul(u, x, accumulate=False, stream=s)
    s.synchronize()
    assert torch.equal(u, ref)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        H.mul(u, x, accumulate=False, stream=s)
    for seed in (7, 8):
        x.copy_(vectors(2500, 1, dtype, seed))
        ref = H @ x
        u.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(u, ref)
    H.free()


def test_low_rank_matrix_columns():
    """Matrices without transfers (one leaf stage, then both parts): one to eight
    columns against the dense product, FP64 to 1e-13 relative."""
    rng = np.random.default_rng(0)
    A = rng.standard_normal((300, 300))
    U, V, s = rng.standard_normal((300, 6)), rng.standard_normal((300, 6)), rng.random(6) + 1

    def dev(a):
        return torch.tensor(np.ascontiguousarray(a.T), device="cuda").t()
    H = hm.HierarchicalMatrix(2, 2)
    H[hm.Block(1), hm.Block(1)] = dev(A)
    H[hm.Block(1), hm.Block(2)] = hm.LowRankMatrix(dev(U), torch.tensor(s, device="cuda"), dev(V))
    H[hm.Block(2), hm.Block(1)] = hm.LowRankMatrix(dev(V), torch.tensor(s, device="cuda"), dev(U))
    H[hm.Block(2), hm.Block(2)] = dev(A.T)
    D = np.block([[A, (U * s) @ V.T], [(V * s) @ U.T, A.T]])
    for k in (1, 2, 4, 7, 8, 9):
        X = rng.standard_normal((600, k))
        got = (H @ (dev(X)[:, 0].contiguous() if k == 1 else dev(X))).cpu().numpy().reshape(600, -1)
        assert np.linalg.norm(got - D @ X) <= 1e-13 * np.linalg.norm(D @ X)
    with pytest.raises(IndexError):
        H @ torch.zeros(599, device="cuda", dtype=torch.float64)

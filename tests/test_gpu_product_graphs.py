"""Products that run as a CUDA graph from their third call on: the same bits as the
first (plain) call, whatever changes between the calls: the vectors' buffers, the
number of right-hand sides (more forms than are kept, scratch that grows), accumulate,
strides, options, streams, threads, a capture by the caller."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import hierarchicalmatrices as hm  # noqa: E402

DT = {"f32": (np.float32, torch.float32), "f64": (np.float64, torch.float64), "df64": ("df64", torch.float64)}


@pytest.fixture(scope="module", params=["f32", "f64", "df64"])
def mat(request):
    n = 30011
    rng = np.random.default_rng(3)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    dt, tdt = DT[request.param]
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=dt)
    yield n, tdt, H
    H.free()


def columns(k, n, tdt, seed=0):
    g = torch.Generator("cuda").manual_seed(100 * seed + k)
    return torch.randn(k, n, device="cuda", dtype=tdt, generator=g).t()


@pytest.mark.parametrize("k", [1, 2, 3, 8, 9, 20])
def test_changing_buffers(mat, k):
    n, tdt, H = mat
    keep = []
    for accumulate in (False, True):
        for seed in range(7):
            B, U0 = columns(k, n, tdt, seed), columns(k, n, tdt, 50 + seed)
            U = U0.clone()
            H.mul(U, B, accumulate=accumulate)
            H.set_overlap(1)                             # another form: its own count of calls
            V = U0.clone()
            H.mul(V, B, accumulate=accumulate)
            H.set_overlap(True)
            keep += [B, U]                               # every call on new buffers
            assert torch.equal(U, V)
    assert H.device_status() == 0


def test_many_forms_and_growing_scratch(mat):
    n, tdt, H = mat
    ks = [1, 3, 2, 5, 9, 4, 12, 16, 1, 24, 6, 3, 1]      # more forms than are kept
    refs = {k: H @ columns(k, n, tdt) for k in set(ks)}
    for _ in range(3):
        for k in ks:
            for _ in range(2):
                assert torch.equal(H @ columns(k, n, tdt), refs[k])
    strided = torch.zeros(3, 2 * n, device="cuda", dtype=tdt)
    for _ in range(5):
        U = strided[:, :n].t()                           # another leading dimension
        H.mul(U, columns(3, n, tdt), accumulate=False)
        assert torch.equal(U, refs[3])


def test_options_are_followed(mat):
    n, tdt, H = mat
    B = columns(1, n, tdt)
    ref = H @ B
    for _ in range(4):
        assert torch.equal(H @ B, ref)
    H.set_near_kernel("stream")
    streamed = [H @ B for _ in range(5)]
    H.set_near_kernel("auto")
    for s in streamed[1:]:
        assert torch.equal(s, streamed[0])
    for pdl in (False, True):
        H.set_pdl(pdl)
        for _ in range(4):
            assert torch.equal(H @ B, ref)


def test_caller_captures(mat):
    n, tdt, H = mat
    B = columns(1, n, tdt)
    U = torch.empty(1, n, device="cuda", dtype=tdt).t()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for _ in range(5):                               # a replayed form on this stream
            H.mul(U, B, accumulate=False, stream=s)
    s.synchronize()
    ref = U.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        H.mul(U, B, accumulate=False, stream=s)
    for _ in range(3):
        U.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(U, ref)
    with torch.cuda.stream(s):
        U.zero_()
        H.mul(U, B, accumulate=False, stream=s)
    s.synchronize()
    assert torch.equal(U, ref)


def test_streams_and_threads(mat):
    n, tdt, H = mat
    cases = [(k, columns(k, n, tdt)) for k in (1, 3, 9)]
    refs = {k: H @ B for k, B in cases}
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for rep in range(8):
                    k, B = cases[(rep + i) % len(cases)]
                    U = torch.empty(k, n, device="cuda", dtype=tdt).t()
                    for _ in range(4):
                        H.mul(U, B, accumulate=False, stream=s)
                    s.synchronize()
                    if not torch.equal(U, refs[k]):
                        errors.append((i, rep, k))
        except Exception as e:                           # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert H.device_status() == 0


def test_transposed_and_gradients():
    n = 20000
    rng = np.random.default_rng(5)
    x, y = (np.sort(rng.random(n))[::-1].copy() for _ in range(2))
    H = hm.KernelMatrix(hm.cauchykernel, x, y, 1.0, 0.0, 1.0, 0.0, dtype=np.float32)
    w, t = torch.randn(2, n, device="cuda")
    first = H.loss_and_grad(w, t)
    for _ in range(6):
        again = H.loss_and_grad(w.clone(), t.clone())
        assert again[0] == first[0]
        for a, b in zip(again[1:], first[1:]):
            assert torch.equal(a, b)
    H.free()

"""Device calls recorded into a CUDA graph, whose kernels start while the one before them runs: a replay on new
windows gives the bits of a direct call.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("mode", ["plain", "chosen"])
@pytest.mark.parametrize("lmax", [3, 33, 530])
@pytest.mark.parametrize("spins", [(0,), (2, 3), (0, 1, 2, 3)])
def test_replay_on_new_windows(mode, lmax, spins):
    from powerspectra_gpu import Context, synthetic as syn
    n, nW = lmax + 1, 2 * lmax + 1
    Ws = [np.stack([syn.mask_spectrum(nW, 0.5, nW / 3.0, seed=10 * k + s) for s in spins]) for k in range(2)]
    ctx = Context(0)
    dW = torch.tensor(Ws[0], device="cuda")
    M = torch.zeros((len(spins), n, n), dtype=torch.float64, device="cuda")

    def call():
        ctx.mcm_multi_device({s: dW[i].data_ptr() for i, s in enumerate(spins)}, nW, 0, lmax,
                             {s: M[i].data_ptr() for i, s in enumerate(spins)}, n, mode=mode)

    s = torch.cuda.Stream()
    ctx.set_stream(s.cuda_stream)
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        want = []
        for W in Ws[::-1]:
            dW.copy_(torch.tensor(W))
            call()
            want.append(M.clone())
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call()
        for W, w in zip(Ws[::-1] + Ws, want + want[::-1]):
            dW.copy_(torch.tensor(W))
            M.zero_()
            g.replay()
            s.synchronize()
            assert bool((M == w).all())

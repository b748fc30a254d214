"""Lifetime of a store's memory: a store may be freed while work on it is still
pending, while another thread captures a graph, and (the differentiable path)
on any stream, and the next one of its size takes nothing away from it."""
import threading

import numpy as np
import pytest

from gpumatting_b200 import api, autograd
from gpumatting_b200.synth import make_problem
from tests.gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def _inputs(W, H, seed=0):
    torch = torch_cuda()
    g = torch.Generator("cuda").manual_seed(seed)
    img = (torch.rand((H, W, 3), generator=g, device="cuda") * 255).to(torch.uint8)
    return img, torch.full((H, W), 255, dtype=torch.uint8, device="cuda")


def test_free_during_another_threads_capture():
    """A free is none of another thread's (thread-local) capture's business: the
    capture ends well, its graph runs, and the freeing thread's next call does
    too."""
    torch = torch_cuda()
    img, scr = _inputs(64, 48)
    st, other = (api.LevinStore(64, 48, "fp16") for _ in range(2))
    st.assemble(img, scr)
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    began, freed, errors = threading.Event(), threading.Event(), []

    def capture():
        try:
            graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.stream(stream):
                graph.capture_begin(capture_error_mode="thread_local")
                x.add_(1.0)
                began.set()
                freed.wait(60)
                x.add_(1.0)
                graph.capture_end()
            graph.replay()
            torch.cuda.synchronize()
        except Exception as e:  # noqa: BLE001 -- reported by the test's thread
            errors.append(e)
            began.set()

    t = threading.Thread(target=capture)
    t.start()
    began.wait(60)
    try:
        del st
        other.assemble(img, scr)
    finally:
        freed.set()
        t.join()
    assert not errors, errors
    torch.cuda.synchronize()
    assert bool((x == 2.0).all())


@pytest.mark.parametrize("W,H", [(256, 200), (1000, 800)])  # either side of 64 MiB
def test_free_with_work_pending(W, H):
    """Products of a store that is freed behind them, while a store of its size is
    made and assembled on another stream: the bits of an undisturbed product."""
    torch = torch_cuda()
    img, scr = _inputs(W, H, 1)
    img2, scr2 = _inputs(W, H, 2)
    x = torch.rand((H, (W + 3) // 4 * 4), device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    want = api.LevinStore(W, H, "fp16").assemble(img, scr).apply(x)
    side, ys = torch.cuda.Stream(), [torch.empty_like(x) for _ in range(50)]
    torch.cuda.synchronize()
    for _ in range(3):
        st = api.LevinStore(W, H, "fp16").assemble(img, scr)
        for y in ys:
            st.apply(x, y)
        del st
        with torch.cuda.stream(side):
            nxt = api.LevinStore(W, H, "fp16").assemble(img2, scr2)
        torch.cuda.synchronize()
        assert all(torch.equal(y[:, :W], want[:, :W]) for y in ys)
        del nxt


@pytest.mark.parametrize("W,H,prec", [(97, 61, "fp16"), (64, 33, "fp32"), (1000, 800, "bf16")])
def test_gradients_on_two_streams_with_recycled_stores(W, H, prec):
    """Steps on two streams in turn, each step's store going back before the
    next: the bits of the same steps one after another on one stream, and of a
    store of api.LevinStore."""
    torch = torch_cuda()
    probs = [make_problem(W, H, k) for k in range(2)]
    data = [(torch.from_numpy(p.image.astype(np.float32) / 255.0).cuda(), torch.from_numpy(p.gamma.astype(np.float32)).cuda(),
             torch.from_numpy(p.s.astype(np.float32)).cuda()) for p in probs]

    def step(k):
        image, gamma, s = data[k]
        image, gamma = image.clone().requires_grad_(), gamma.clone().requires_grad_()
        alpha = autograd.levin_matte(image, gamma, s, eps=1e-3, precision=prec)
        ((alpha - 0.25) ** 2).mean().backward()
        return alpha.detach(), image.grad, gamma.grad

    want = [step(k) for k in range(2)]
    im4 = torch.zeros((H, W, 4), device="cuda")
    im4[..., :3] = data[0][0]
    plain = torch.full((H, W), 0.5, device="cuda")
    api.LevinStore(W, H, prec).assemble(im4, gamma_map=data[0][1], s_map=data[0][2], eps=1e-3).solve(
        plain, "mg", rtol=1e-6, max_iters=5000)
    assert torch.equal(plain, want[0][0])
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for i in range(6):
        with torch.cuda.stream(streams[i % 2]):
            got = step(i % 2)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want[i % 2]))

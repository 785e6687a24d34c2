"""The gradient kernel at the edges of its row tiles (16 rows a warp, 64 a CTA) and where a CTA takes several
tiles, called twice (the second call finds the gradients empty), against a restatement in 64 bits that
rounds to halves where the kernel does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _half(a):
    return a.astype(np.float16).astype(np.float64)


def _gradients(p, x, y):
    p, x, y = p.astype(np.float64), x.astype(np.float64), y.astype(np.float64)
    w1, b1, w2, b2, w3, b3 = _half(p[:2048]).reshape(32, 64), p[2048:2112], _half(p[2112:6208]).reshape(64, 64), p[6208:6272], p[6272:6336], p[6336]
    h1 = np.maximum(x @ w1 + b1, 0)
    h2 = np.maximum(_half(h1) @ w2 + b2, 0)
    dz = (1 / (1 + np.exp(-(h2 @ w3 + b3))) - y) / len(y)
    d2 = np.outer(dz, w3) * (h2 > 0)
    d1 = (_half(d2) @ w2.T) * (h1 > 0)
    return np.concatenate([(x.T @ _half(d1)).ravel(), d1.sum(0), (_half(h1).T @ _half(d2)).ravel(), d2.sum(0), h2.T @ dz, [dz.sum()]])


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 129, 2 * 148 * 64 + 1])
def test_gradients_at_tile_edges(vf, n):
    import torch

    from vfwater import proposal

    mlp = proposal.MLP(seed=4)
    rng = np.random.default_rng(n)
    x = (rng.random((n, 32)) * (rng.random((n, 32)) < 0.5)).astype(np.float16)
    # labels of one row in 64 only, so that the gradients of many rows do not cancel; halves of 1/n keep
    # their precision down to n = 2^14 / 2^-14 (below 6e-5 their step is 2^-24)
    y = (rng.random(n) < 1 / 64).astype(np.float32)
    ref = _gradients(mlp.params(), x, y)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    # the sums differ in the order of fp32 additions, and an operand next to a rounding boundary by a half's
    # step: 2^-10 of its value, or 2^-24 of each of the n rows' products with values up to 4
    tol = 2.0**-10 * np.abs(ref).max() + 4 * n * 2.0**-24 * 2.0**-5
    for _ in range(2):
        assert np.abs(mlp.grads(xd, yd) - ref).max() <= tol
    mlp.close()


def test_a_refused_call_leaves_the_handle_as_it_was():
    """Gradients wait for the host, which a stream under capture refuses: the call fails, and the next one is right
    (in a process of its own, for the broken capture)."""
    import subprocess
    import sys
    from pathlib import Path

    code = """
import numpy as np, torch
import __graft_entry__ as ge
vf = ge.load_package()
from vfwater import proposal
mlp = proposal.MLP(seed=4)
x = torch.rand(200, 32, device="cuda").half()
y = (torch.rand(200, device="cuda") < 0.5).float()
want = mlp.grads(x, y)
graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
refused = []
try:
    with torch.cuda.graph(graph, stream=stream):
        for call in (lambda: mlp.grads(x, y, stream=stream.cuda_stream), lambda: mlp.train_step(x, y, 0.0, stream=stream.cuda_stream, want_loss=True)):
            try:
                call()
            except vf.VfError:
                refused.append(1)
except RuntimeError:
    pass
assert len(refused) == 2, refused
torch.cuda.synchronize()
for _ in range(2):
    assert np.allclose(mlp.grads(x, y), want, rtol=1e-5, atol=1e-9)
print("ok")
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("rows", [1, 300, 100000])  # fewer rows than slots, more than the atlas holds
def test_staging_counts_rows_and_changes_nothing(vf, ring, rows):
    import torch

    from vfwater import proposal

    if ring:
        w = vf.World.ring(4, 64)
        chunk = vf.World(128, 64, 128)
        chunk.fill_box(0, 0, 0, 127, 7, 127, 3)
        for cx in (-1, 0):
            w.ring_paste(chunk, cx, 0)
        w.fill_box(-20, 8, 40, 19, 30, 59, 5)
        box = (-24, 7, 36, 23, 34, 63)
    else:
        w = vf.World(61, 43, 77)  # bricks that reach past the world on every side
        w.fill_box(0, 0, 0, 60, 3, 76, 3)
        w.fill_box(30, 4, 40, 60, 30, 76, 5)
        box = (0, 0, 0, 60, 42, 76)
    sim = vf.FluidSim(w, atlas_bricks=2000)
    sim.wake(*box)
    sim.tick(5)
    if ring:
        sim.ring_evict(0, 0)
    before = sim.digest()
    p = torch.rand(rows, device="cuda")
    p[0] = 0.5
    n = min(rows, max(2000, sim.stats().atlas_used + 64))
    staged = proposal.stage(sim, p, 0.5)
    assert staged <= int((p >= 0.5).sum()) and (rows > 1000 or staged == int((p[:n] >= 0.5).sum()))
    assert sim.digest() == before
    sim.tick(2)
    sim.close()

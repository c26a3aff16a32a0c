"""The fused layer, gradient and reduction kernels of the warm-start MLP at their edges, against
oracle/mlp_oracle.py: one point, slots that begin and end inside a tile or a backward block,
one-point slots, more 128-point tiles than SMs with a partial last one, and a handle reused with
fewer points. Tolerances as in test_gpu_mlp.py (BF16 rounding flips)."""
import numpy as np
import pytest

from test_gpu_mlp import _mlp_case

pytestmark = pytest.mark.gpu

CASES = {"one point": (0, 1), "inside a block": (0, 63, 64, 65, 129), "one-point slots": tuple(range(151)),
         "block edges": (0, 64, 128, 192, 256), "many tiles": (0, 5000, 19000, 153 * 128 + 77), "one slot": (0, 700)}


def test_forward_and_gradient_match_oracle(cuda):
    import torch

    from oracle import mlp_oracle as mo
    from plugin_navierstokes_gb300.warm_start import CoordinateMLP

    m = CoordinateMLP(max_points=20000, max_slots=160)
    off, _ = mo.offsets()
    for name in ("many tiles", "one point", "inside a block", "one-point slots", "block edges", "one slot"):
        slots = CASES[name]
        P = slots[-1]
        p, xy, sp, cond, target = _mlp_case(P, P, slots)
        m.set_params(p)
        txy = torch.from_numpy(xy).to(cuda)
        out = torch.empty((P, 3), dtype=torch.float32, device=cuda)
        m.forward(txy, sp, cond, out)
        ref, _ = mo.forward(p, xy, sp, cond, use_bf16=True)
        e = np.linalg.norm(out.double().cpu().numpy() - ref) / np.linalg.norm(ref)
        assert e < 2e-3, (name, e)
        grad = torch.full((m.num_params,), float("nan"), dtype=torch.float32, device=cuda)
        loss = m.loss_grad(txy, sp, cond, torch.from_numpy(target).to(cuda), grad)
        lref, gref = mo.loss_grad(p, xy, sp, cond, target, use_bf16=True)
        assert abs(loss - lref) <= 1e-3 * lref, name
        g = grad.double().cpu().numpy()
        for key, (o, size) in off.items():
            r = gref[o:o + size]
            e = np.linalg.norm(g[o:o + size] - r) / max(np.linalg.norm(r), 1e-30)
            assert e < 1e-2, (name, key, e)
        again = torch.empty_like(grad)
        assert m.loss_grad(txy, sp, cond, torch.from_numpy(target).to(cuda), again) == loss
        assert torch.equal(grad, again), name


def test_predict_in_chunks_gives_the_same_state(cuda):
    """A prediction split into chunks of whole slots equals one that fits the capacity, bit for bit."""
    import torch

    from plugin_navierstokes_gb300.warm_start import CoordinateMLP

    slots = (0, 700, 701, 1500, 2000)
    p, xy, sp, cond, _ = _mlp_case(3, slots[-1], slots)
    lid = np.linspace(0.5, 2.0, 4).astype(np.float32)
    states = []
    for cap in (2048, 800):
        m = CoordinateMLP(max_points=cap, max_slots=4)
        m.set_params(p)
        u = torch.empty(slots[-1] * 3, dtype=torch.float64, device=cuda)
        m.predict(torch.from_numpy(xy).to(cuda), sp, cond, lid, u)
        states.append(u)
    assert torch.isfinite(states[0]).all() and torch.equal(states[0], states[1])

"""Host branches of a call: calls that need no autograd Function, batches run
whole and split when an allocation fails, forward-mode levels and repeated
argument devices."""
import numpy as np
import pytest
import torch

import jaqsi_b200 as jq
from jaqsi_b200 import simulation as sim

pytestmark = pytest.mark.gpu


def _circuit(p):
    for w in range(3):
        jq.RY(p[w], wires=w)
    for w in range(3):
        jq.CX(wires=[w, (w + 1) % 3])


OBS = [jq.PauliZ(0), jq.PauliZ(2)]


@pytest.mark.parametrize("noisy", [False, True])
def test_reverse_call_halves_its_batch_when_memory_runs_out(monkeypatch, noisy):
    def circuit(p):
        _circuit(p)
        if noisy:
            jq.DepolarizingChannel(0.1, wires=0)

    script = jq.Script(circuit, n_qubits=3)
    base = torch.rand(7, 3, generator=torch.Generator().manual_seed(1), dtype=torch.float64)
    grads, seen = [], []
    whole = sim._grad_launch_whole

    def limited(plan, out_type, batch, *rest):
        seen.append(batch)
        if batch > 2:
            raise torch.OutOfMemoryError("test")
        return whole(plan, out_type, batch, *rest)

    for patched in (False, True):
        if patched:
            monkeypatch.setattr(sim, "_grad_launch_whole", limited)
        p = base.clone().requires_grad_(True)
        script.execute("expval", OBS, args=(p,), in_axes=(0,)).sum().backward()
        grads.append(p.grad.clone())
    assert seen[0] == 7 and max(b for b in seen if b <= 2) == 2
    torch.testing.assert_close(grads[0], grads[1], atol=1e-14, rtol=0)


def test_small_batches_run_whole_and_fall_back_to_chunks(monkeypatch):
    script = jq.Script(_circuit, n_qubits=3)
    p = torch.rand(6, 3, generator=torch.Generator().manual_seed(2), dtype=torch.float64)
    want = script.execute("expval", OBS, args=(p,), in_axes=(0,))
    run, batches = sim.run_plan, []

    def limited(plan, out_type, batch, *rest):
        batches.append(batch)
        if batch > 4:
            raise torch.OutOfMemoryError("test")
        return run(plan, out_type, batch, *rest)

    monkeypatch.setattr(sim, "run_plan", limited)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (1, 0))  # chunks of one instance
    got = script.execute("expval", OBS, args=(p,), in_axes=(0,))
    assert batches == [6] + [1] * 6
    torch.testing.assert_close(got, want, atol=0, rtol=0)


def test_forward_mode_levels_and_saved_tensor_hooks_still_see_the_function():
    script = jq.Script(_circuit, n_qubits=3)
    x = torch.tensor([0.3, 0.7, 1.1], dtype=torch.float64)
    v = torch.tensor([0.2, -1.0, 0.5], dtype=torch.float64)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x, v)
        out = script.execute("expval", OBS, args=(dual,))
        tangent = torch.autograd.forward_ad.unpack_dual(out).tangent
    h = 1e-6
    fd = (script.execute("expval", OBS, args=(x + h * v,)) - script.execute("expval", OBS, args=(x - h * v,))) / (2 * h)
    assert tangent is not None
    np.testing.assert_allclose(tangent.cpu().numpy(), fd.cpu().numpy(), atol=1e-8)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t, lambda t: t):
        y = x.clone().requires_grad_(True)
        out = script.execute("expval", OBS, args=(y,))
    out.sum().backward()
    assert packed and y.grad is not None
    # a second derivative is refused, not silently zero
    y = x.clone().requires_grad_(True)
    (g,) = torch.autograd.grad(script.execute("expval", OBS, args=(y,)).sum(), y, create_graph=True)
    with pytest.raises(RuntimeError):
        g.sum().backward()

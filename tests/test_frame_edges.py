"""Edges of the frame and Pauli plans (csrc/frame.h): inputs and sizes at which
they branch, against the general passes (an explicit |0..0> start or
``expval_only = 1``), against single calls, or against the oracle.

Tolerances, set before the first run, are those of the other parity tests:
1e-10 (complex128) and 1e-5 (complex64), absolute, times the weight of the
cotangents.
"""
import numpy as np
import pytest
import torch

import jaqsi_b200 as jq
from jaqsi_b200 import _lib as L
from jaqsi_b200 import simulation as sim
from jaqsi_b200 import workloads as wl
from oracle import sim_np as O
from tests.helpers import obs_records, to_records

pytestmark = pytest.mark.gpu
TOL = {torch.complex64: 1e-5, torch.complex128: 1e-10}


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [5, 6])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("gate", [jq.RZ, jq.RY])
def test_noisy_values_of_an_angle_that_is_not_finite(n, bad, gate, dtype):
    """One such angle leaves the density matrix without a finite entry: every
    value and every gradient of its sample is NaN, those of the others are not."""

    def circuit(p):
        gate(p[0], wires=0)
        for w in range(1, n):
            jq.RY(p[w], wires=w)
        jq.DepolarizingChannel(0.1, wires=1)

    params = torch.full((3, n), 0.3, dtype=torch.float64)
    params[1, 0] = bad
    params.requires_grad_(True)
    script = jq.Script(circuit, n_qubits=n)
    ev = script.execute("expval", [jq.PauliZ(w) for w in range(n)], args=(params,), in_axes=(0,), dtype=dtype)
    ev.sum().backward()
    assert torch.isnan(ev[1]).all() and torch.isnan(params.grad[1]).all()
    assert torch.isfinite(ev[[0, 2]]).all() and torch.isfinite(params.grad[[0, 2]]).all()
    assert torch.equal(ev[0], ev[2])


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("n", [5, 6])
def test_noisy_gradients_of_a_cotangent_that_is_not_finite(n, bad, dtype):
    """Every gradient of that sample is NaN, also of gates the observable's word does
    not reach; those of the others are not."""

    def circuit(p):
        for w in range(n):
            jq.RY(p[w], wires=w)
            jq.DepolarizingChannel(0.1, wires=w)

    params = torch.full((3, n), 0.3, dtype=torch.float64, requires_grad=True)
    script = jq.Script(circuit, n_qubits=n)
    ev = script.execute("expval", [jq.PauliZ(w) for w in range(n)], args=(params,), in_axes=(0,), dtype=dtype)
    ct = torch.ones_like(ev)
    ct[1, 2] = bad
    ev.backward(ct)
    assert torch.isnan(params.grad[1]).all()
    assert torch.isfinite(params.grad[[0, 2]]).all() and torch.equal(params.grad[0], params.grad[2])


@pytest.mark.parametrize("n", [9, 10, 11, 12, 13, 15])
def test_frame_cotangent_sums_of_small_states_are_float64(n):
    """Complex64 states below 2^16 amplitudes.  Wire a starts in |+> and has no gate,
    the others are turned into |+>, amplitudes exact but for a factor common to
    all.  Where z_a = 1 the words z_x z_y (1 + z_a) / 2 leave every gradient zero in
    terms of size 1; where z_a = -1, 2^-28 z_w (1 - z_a) / 2 has terms of size 2^-28,
    which float32 sums over both lose and float64 sums hold to 2^-24."""
    rng = np.random.default_rng(n)
    parity = jq.build_parity_observable
    for _ in range(100):
        a, x, y, w = (int(v) for v in rng.choice(n, 4, replace=False))
        script = jq.Script(lambda p: [jq.RY(p[k], wires=k) for k in range(n) if k != a] and None, n_qubits=n)
        start = torch.zeros(2**n, dtype=torch.complex64)
        start[0] = start[1 << (n - 1 - a)] = 0.5**0.5
        obs = [parity([x, y]), parity([a, x, y]), jq.PauliZ(w), parity([a, w])]
        params = torch.full((n,), np.pi / 2, dtype=torch.float64, requires_grad=True)
        ev = script.execute("expval", obs, args=(params,), initial_state=start, dtype=torch.complex64)
        ct = torch.tensor([0.5, 0.5, 2.0**-29, -(2.0**-29)], device=ev.device, dtype=torch.float64)
        (ev.to(torch.float64) @ ct).backward()
        want = np.zeros(n)
        want[w] = -(2.0**-29)
        np.testing.assert_allclose(params.grad.numpy(), want, atol=TOL[torch.complex64] * 2.0**-29, rtol=0,
                                   err_msg=f"{a} {x} {y} {w}")


@pytest.mark.parametrize("n", [5, 6, 7])
def test_pauli_cotangent_sums_of_small_states_are_float64(n):
    """Complex64 coefficients below 2^16: wires b, c, d stay in |0>, so that z_w z_b -
    z_w z_c + 2^-28 z_w z_d has the gradient of 2^-28 z_w, whose terms in a sum
    over coefficients are 1, -1 and 2^-28."""
    parity = jq.build_parity_observable

    def circuit(p):
        jq.RY(p[0], wires=0)
        jq.AmplitudeDamping(0.1, wires=0)

    script = jq.Script(circuit, n_qubits=n)
    want = -(2.0**-28) * 0.9 * np.sin(0.7)
    for b in range(1, n):
        for c in range(1, n):
            for d in range(1, n):
                if len({b, c, d}) < 3:
                    continue
                p = torch.tensor([0.7], dtype=torch.float64, requires_grad=True)
                ev = script.execute("expval", [parity([0, b]), parity([0, c]), parity([0, d])], args=(p,),
                                    dtype=torch.complex64)
                ct = torch.tensor([1.0, -1.0, 2.0**-28], device=ev.device, dtype=torch.float64)
                (ev.to(torch.float64) @ ct).backward()
                np.testing.assert_allclose(p.grad.numpy(), [want], rtol=TOL[torch.complex64], err_msg=f"{b} {c} {d}")


def _noisy_plans(n, layers, noise, obs, dtype):
    """A noisy circuit on the general passes and on Pauli coefficients."""
    with jq.recording() as tape:
        wl.noisy_ansatz(n, layers, np.zeros((layers, n, 3)), noise, noise)
    lw = sim.lower_tape(tape, n)
    specs, _ = sim._lower_obs(obs, n)
    statics = [st[:10] + (1,) + st[11:] if st[3] >= 0 else st for st in lw.statics]  # every angle trainable
    return [sim.Plan(statics, specs, n, L.JQ_DENSITY, dtype, {"expval_only": e}) for e in (1, 2)]


def _backward(plan, angles, ct, with_grad):
    batch = angles.shape[0]
    grad = torch.empty((batch, plan.n_angles), dtype=torch.float64, device="cuda")
    ws = torch.full((plan.workspace_bytes(batch, with_grad),), 255, dtype=torch.uint8, device="cuda")  # NaNs
    L.check(plan._lib.jq_backward(plan.handle, batch, sim._ptr(angles), None, None, 0, L.JQ_OUT_EXPVAL, sim._ptr(ct),
                                  None, sim._ptr(grad), None, None, sim._ptr(ws), ws.numel(), sim._stream()))
    return grad.cpu().numpy()


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,layers,batch", [(6, 40, 2), (6, 80, 1), (7, 40, 1), (7, 60, 2), (9, 20, 1)])
def test_segments_of_the_pauli_reverse_pass(n, layers, batch, dtype):
    """More passes than the least workspace holds states: the inputs of a segment are
    recomputed from its checkpoint.  Every gradient, against the call that keeps
    all inputs (the same kernels on the same values: only the order of float64
    additions differs) and against the general passes."""
    rng = np.random.default_rng(n * layers)
    obs = [jq.PauliZ(0), jq.PauliX(n - 1), jq.PauliZ(2)]
    general, own = _noisy_plans(n, layers, 0.001, obs, dtype)
    half = own.state_elems * batch * (4 if dtype == torch.complex64 else 8)
    assert own.info["n_passes_fwd"] > own.workspace_bytes(batch, 2) // half
    angles = torch.tensor(rng.uniform(0, 2 * np.pi, (batch, own.n_angles)), device="cuda")
    ct = torch.tensor(rng.normal(size=(batch, len(obs))), device="cuda")
    least, roomy = _backward(own, angles, ct, 2), _backward(own, angles, ct, 3)
    np.testing.assert_allclose(least, roomy, atol=1e-13, rtol=0)
    want = _backward(general, angles, ct, 2)
    np.testing.assert_allclose(least, want, atol=TOL[dtype] * np.abs(ct.cpu().numpy()).sum(1).max() * n, rtol=0)
    assert np.abs(want).max() > 1e-3


def test_reverse_call_takes_less_where_memory_is_short(monkeypatch):
    """The larger workspace does not fit: the call runs in the smaller one."""
    n, layers = 7, 40
    script = jq.Script(lambda a: wl.noisy_ansatz(n, layers, a, 0.001, 0.001), n_qubits=n)
    base = torch.rand(layers, n, 3, generator=torch.Generator().manual_seed(3), dtype=torch.float64) * 6
    given, make = [], sim._workspace

    def limited(nbytes, dev):
        given.append(nbytes)
        if len(given) == 1:
            raise torch.OutOfMemoryError("test")
        return make(nbytes, dev)

    grads = []
    for patched in (False, True):
        if patched:
            monkeypatch.setattr(sim, "_workspace", limited)
        p = base.clone().requires_grad_(True)
        script.execute("expval", [jq.PauliZ(0)], args=(p,)).sum().backward()
        grads.append(p.grad)
    assert len(given) == 2 and given[1] < given[0]
    torch.testing.assert_close(grads[0], grads[1], atol=1e-13, rtol=0)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [9, 13])
def test_sweeps_of_a_frame_plan_follow_one_another(n, dtype):
    """jq_sweep applies the circuit to amplitudes at their own indices, also under
    expval_only = 2: twice from a random state, against the oracle."""
    rng = np.random.default_rng(n)

    def circuit(p):
        for l in range(2):
            for w in range(n):
                jq.Rot(p[l, w, 0], p[l, w, 1], p[l, w, 2], wires=w)
            if l == 0:
                for w in range(n):
                    jq.CX(wires=[w, (w + 1) % n])
                jq.PauliX(wires=2)
                jq.SWAP(wires=[0, n - 1])

    base = torch.tensor(rng.uniform(0, 2 * np.pi, (2, n, 3)))
    script = jq.Script(circuit, n_qubits=n)
    plan = sim.get_plan(sim.lower_tape(script.record(base), n), *sim._lower_obs([jq.PauliZ(0)], n), n,
                        L.JQ_STATEVECTOR, dtype)
    psi = rng.normal(size=2**n) + 1j * rng.normal(size=2**n)
    psi /= np.linalg.norm(psi)
    angles = base.reshape(-1).to("cuda")
    state = torch.tensor(psi, dtype=dtype, device="cuda")
    ws = torch.empty(plan.workspace_bytes(1), dtype=torch.uint8, device="cuda")
    recs = to_records(script.record(base))
    for _ in range(2):
        L.check(plan._lib.jq_sweep(plan.handle, 1, sim._ptr(angles), None, sim._ptr(state), sim._ptr(ws), ws.numel(),
                                   sim._stream()))
        psi = O.simulate_pure(recs, n, psi)
        np.testing.assert_allclose(state.cpu().numpy(), psi, atol=TOL[dtype], rtol=0)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_sweeps_of_a_pauli_plan_work_on_matrix_entries(dtype):
    n, layers = 5, 2
    rng = np.random.default_rng(3)
    obs = [jq.PauliZ(0)]
    general, own = _noisy_plans(n, layers, 0.02, obs, dtype)
    angles = torch.tensor(rng.uniform(0, 2 * np.pi, own.n_angles), device="cuda")
    a = rng.normal(size=(2**n, 2**n)) + 1j * rng.normal(size=(2**n, 2**n))
    rho = a @ a.conj().T
    rho = torch.tensor(rho / np.trace(rho), dtype=dtype, device="cuda")
    got = []
    for plan in (general, own):
        state = rho.clone()
        ws = torch.empty(plan.workspace_bytes(1), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            L.check(plan._lib.jq_sweep(plan.handle, 1, sim._ptr(angles), None, sim._ptr(state), sim._ptr(ws), ws.numel(),
                                       sim._stream()))
        got.append(state.cpu().numpy())
    np.testing.assert_allclose(got[1], got[0], atol=TOL[dtype], rtol=0)
    assert abs(np.trace(got[1]) - 1) < 10 * TOL[dtype]


def _values_and_gradients(plan, angles, rows):
    """Expectation values and the gradients of their weighted sum, `rows` instances a call."""
    values, grads = [], []
    for a in angles.split(rows):
        state, out = sim._forward_launch(plan, L.JQ_OUT_EXPVAL, a.shape[0], 0, a, None, None)
        ct = torch.linspace(0.5, 1.5, plan.n_obs, dtype=torch.float64, device="cuda").expand(a.shape[0], -1)
        values.append(out)
        grads.append(sim._grad_launch(plan, L.JQ_OUT_EXPVAL, a.shape[0], 0, (True, False, False), a, None, None, state, ct)[0])
    return torch.cat(values), torch.cat(grads)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,batch,noisy", [(9, 6000, False), (10, 5000, False), (12, 1300, False), (13, 600, False),
                                           (16, 80, False), (5, 5000, True), (6, 1300, True), (8, 80, True)])
def test_batches_of_more_tiles_than_fit_at_once(n, batch, noisy, dtype):
    """A CTA goes from one instance's tiles to the next one's: new gate tables, sums
    handed over.  Every instance has angles of its own; a call on eight of them
    has a CTA a tile.  The kernels do the same arithmetic on a tile in both, so
    that only the order of float64 additions differs."""
    layers = 2
    with jq.recording() as tape:
        if noisy:
            wl.noisy_ansatz(n, layers, np.zeros((layers, n, 3)), 0.01, 0.02)
        else:
            wl.rot_ring(n, layers, np.zeros((layers, n, 3)))
    lw = sim.lower_tape(tape, n)
    obs = [jq.PauliZ(w) for w in range(n)]
    specs, _ = sim._lower_obs(obs, n)
    statics = [st[:10] + (1,) + st[11:] if st[3] >= 0 else st for st in lw.statics]  # every angle trainable
    mode = L.JQ_DENSITY if noisy else L.JQ_STATEVECTOR
    general, plan = [sim.Plan(statics, specs, n, mode, dtype, {"expval_only": e}) for e in (1, 2)]
    assert plan.info != general.info
    bits = 2 * n if noisy else n
    tile = bits if bits <= 10 or (bits == 12 and not noisy) else 11
    most = torch.cuda.get_device_properties(0).multi_processor_count * min(32, 2048 // (1 << (tile - 4)))
    assert batch << (bits - tile) > most
    angles = torch.tensor(np.random.default_rng(n).uniform(0, 2 * np.pi, (batch, plan.n_angles)), device="cuda")
    for all_at_once, few in zip(_values_and_gradients(plan, angles, batch), _values_and_gradients(plan, angles, 8)):
        torch.testing.assert_close(all_at_once, few, atol=1e-12, rtol=0)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,layers", [(9, 5), (10, 7), (11, 9), (12, 5), (12, 12)])
def test_whole_state_tiles_of_many_stages(n, layers, dtype):
    """States of one tile: more stages than tile flips are kept for, and (the longest)
    more than a pass holds, against the oracle."""
    rng = np.random.default_rng(n * layers)
    base = rng.uniform(0, 2 * np.pi, (layers, n, 3))
    script = jq.Script(lambda a: wl.rot_ring(n, layers, a), n_qubits=n)
    obs = [jq.PauliZ(0), jq.build_parity_observable([1, n - 1])]
    lw = sim.lower_tape(script.record(torch.tensor(base)), n)
    info = sim.get_plan(lw, *sim._lower_obs(obs, n), n, L.JQ_STATEVECTOR, dtype).info
    assert info["n_stages_fwd"] > 8 and info["n_tile_ops_fwd"] == n * layers
    assert info["n_passes_fwd"] == (1 if info["n_stages_fwd"] <= 24 else 2)
    params = torch.tensor(base, requires_grad=True)
    ev = script.execute("expval", obs, args=(params,), dtype=dtype)
    ev.sum().backward()
    want, grad = O.adjoint_grad(to_records(script.record(torch.tensor(base))), n, obs_records(obs), ct=np.ones(2))
    np.testing.assert_allclose(ev.detach().cpu().numpy(), want, atol=TOL[dtype], rtol=0)
    np.testing.assert_allclose(params.grad.numpy().reshape(-1), grad, atol=TOL[dtype] * 2, rtol=0)


def _linear(rng, k):
    """A random invertible 0/1 matrix over GF(2) as columns, and its permutation."""
    while True:
        col = [int(v) for v in rng.integers(1, 1 << k, k)]
        to = [0] * (1 << k)
        for x in range(1 << k):
            for i in range(k):
                if x >> i & 1:
                    to[x] ^= col[i]
        if len(set(to)) == 1 << k:
            return to


def _permuting(rng, k, shift):
    """A gate that takes basis state x to A x ^ b (b = 0 unless `shift`)."""
    to = _linear(rng, k)
    b = int(rng.integers(1 << k)) if shift else 0
    perm = [0] * (1 << k)
    for x, y in enumerate(to):
        perm[y ^ b] = x  # output row r takes input column perm[r]
    m = np.zeros((1 << k, 1 << k), dtype=np.complex128)
    m[np.arange(1 << k), perm] = 1
    return type(f"Perm{k}_{rng.integers(1 << 40)}", (jq.Operation,),
                {"_matrix": m, "_num_wires": k, "is_unitary": True, "_structure": jq.operations.GateStructure(permutation=tuple(perm))})


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,noisy", [(9, False), (12, False), (13, False), (16, False), (5, True), (6, True), (7, True), (8, True)])
def test_every_permutation_that_is_accepted(n, noisy, dtype):
    """Random affine permutations of two to six wires (linear ones of two to four
    on Pauli words) in any wire order, rotations by every generator, constants and
    random Kraus sets, Pauli words with either sign: against the general passes."""
    rng = np.random.default_rng(31 * n + noisy)

    def circuit(p):
        k = 0
        for _ in range(4):
            for w in range(n):
                kind = int(rng.integers(6))
                if kind == 0:
                    jq.Rot(p[k], p[k + 1], p[k + 2], wires=w)
                    k += 3
                elif kind < 4:
                    jq.PauliRot(p[k], "XYZ"[kind - 1], wires=[w])
                    k += 1
                elif kind == 4:
                    jq.H(wires=w)
                    jq.S(wires=w)
                if noisy and rng.integers(2):
                    q, _ = np.linalg.qr(rng.normal(size=(6, 2)) + 1j * rng.normal(size=(6, 2)))
                    jq.QubitChannel([np.sqrt(0.9) * np.eye(2)] + [np.sqrt(0.1) * q[2 * i:2 * i + 2] for i in range(3)], wires=w)
            for _ in range(3):
                size = int(rng.integers(2, 5 if noisy else 7))
                wires = [int(w) for w in rng.choice(n, size, replace=False)]
                _permuting(rng, size, not noisy)(wires=wires)
        for w in range(n):
            jq.RY(p[k + w], wires=w)
        return k + n

    with jq.recording() as tape:
        count = circuit(torch.zeros(16 * n + 16))
    assert count <= 16 * n + 16
    pauli = [np.eye(2), np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]]), np.diag([1.0, -1.0])]
    obs = []
    for _ in range(12):
        wires = [int(w) for w in rng.choice(n, 3, replace=False)]
        m = np.array([[rng.choice([-1.5, 0.5, 2.0])]])
        for _ in wires:
            m = np.kron(m, pauli[int(rng.integers(4)) if noisy else 3 * int(rng.integers(2))])
        obs.append(jq.Hermitian(m, wires=wires, record=False))
    lw = sim.lower_tape(tape, n)
    specs, _ = sim._lower_obs(obs, n)
    statics = [st[:10] + (1,) + st[11:] if st[3] >= 0 else st for st in lw.statics]  # every angle trainable
    mode = L.JQ_DENSITY if noisy else L.JQ_STATEVECTOR
    general, own = [sim.Plan(statics, specs, n, mode, dtype, {"expval_only": e, "jit": 0 if e == 2 else -1}) for e in (1, 2)]
    assert own.info["n_tile_ops_fwd"] != general.info["n_tile_ops_fwd"]  # permutations are none in either
    angles = torch.tensor(rng.uniform(0, 2 * np.pi, (2, own.n_angles)), device="cuda")
    got, want = _values_and_gradients(own, angles, 2), _values_and_gradients(general, angles, 2)
    for g, w in zip(got, want):
        np.testing.assert_allclose(g.cpu().numpy(), w.cpu().numpy(), atol=TOL[dtype] * 2.0 * len(obs), rtol=0)
    assert got[0].abs().max() > 1e-3 and got[1].abs().max() > 1e-3


@pytest.mark.parametrize("n,noisy", [(9, False), (13, False), (5, True), (6, True)])
def test_torch_func_transforms_in_both_representations(n, noisy):
    """jacrev, jvp, vmap and a batched initial state through the plan's own state
    buffers, against one reverse call per value."""
    layers = 2
    body = (lambda a: wl.noisy_ansatz(n, layers, a, 0.01, 0.02)) if noisy else (lambda a: wl.rot_ring(n, layers, a))
    script = jq.Script(body, n_qubits=n)
    obs = [jq.PauliZ(0), jq.PauliZ(n - 1), jq.build_parity_observable([1, 2])]
    p = torch.tensor(np.random.default_rng(n).uniform(0, 2 * np.pi, (layers, n, 3)), device="cuda")

    def f(x):
        return script.execute("expval", obs, args=(x,))

    rows = []
    for o in range(len(obs)):
        x = p.clone().requires_grad_(True)
        rows.append(torch.autograd.grad(f(x)[o], x)[0])
    rows = torch.stack(rows)
    torch.testing.assert_close(torch.func.jacrev(f)(p), rows, atol=1e-12, rtol=0)
    v = torch.randn(p.shape, generator=torch.Generator("cuda").manual_seed(1), device="cuda", dtype=torch.float64)
    value, tangent = torch.func.jvp(f, (p,), (v,))
    torch.testing.assert_close(value, f(p), atol=1e-13, rtol=0)
    torch.testing.assert_close(tangent, (rows * v).sum((1, 2, 3)), atol=1e-11, rtol=0)
    many = torch.stack([p, p + 0.1, 2 * p])
    each = torch.stack([f(x) for x in many])
    torch.testing.assert_close(torch.func.vmap(f)(many), each, atol=1e-13, rtol=0)
    torch.testing.assert_close(script.execute("expval", obs, args=(many,), in_axes=(0,)), each, atol=1e-13, rtol=0)
    grads = torch.func.vmap(torch.func.grad(lambda x: f(x).sum()))(many)
    torch.testing.assert_close(grads[0], rows.sum(0), atol=1e-12, rtol=0)


@pytest.mark.parametrize("n,noisy", [(9, False), (13, False), (6, True)])
def test_threads_on_streams_of_their_own(n, noisy):
    """Four threads, each on its own stream, share a script and its plan from its
    first call on: the results of calls one after the other."""
    import threading

    layers = 2
    body = (lambda a: wl.noisy_ansatz(n, layers, a, 0.01, 0.02)) if noisy else (lambda a: wl.rot_ring(n, layers, a))
    obs = [jq.PauliZ(0), jq.PauliZ(n - 1)]
    params = torch.tensor(np.random.default_rng(n).uniform(0, 2 * np.pi, (4, layers, n, 3)), device="cuda")

    def step(script, k):
        x = params[k].clone().requires_grad_(True)
        value = script.execute("expval", obs, args=(x,))
        return value.detach(), torch.autograd.grad(value.sum(), x)[0]

    shared = jq.Script(body, n_qubits=n)
    got = [[] for _ in range(4)]
    failed = []

    def work(k, stream):
        try:
            with torch.cuda.stream(stream):
                for _ in range(20):
                    got[k].append(step(shared, k))
        except Exception as e:  # pragma: no cover - reported below
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k, torch.cuda.Stream())) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    alone = jq.Script(body, n_qubits=n)
    for k in range(4):
        want = step(alone, k)
        assert len(got[k]) == 20
        for value, grad in got[k]:
            torch.testing.assert_close(value, want[0], atol=1e-13, rtol=0)
            torch.testing.assert_close(grad, want[1], atol=1e-12, rtol=0)

"""Workloads of the circuit-execution path, as a user's program calls it.

A case names a circuit family, its size and what is asked of it.  Three kinds
of call exist, the three that a program makes:

- ``call``: ``Script.execute`` for expectation values, probabilities, a state
  or a density matrix (one parameter set, or ``batch`` sets through
  ``in_axes``).  A ``Script`` is kept between calls, as a program keeps it.
- ``train``: the same call followed by the gradient with respect to the
  parameters, the body of a training step.
- ``uneven``: ``BatchedGradients`` over many circuits of different sizes and
  depths: new angles in, expectation values and gradients out.  The handle is
  kept between steps.

Angles are uniform in [0, 2 pi), the start state is |0..0>; single precision
programs hold float32 parameters, double precision ones float64.
"""
import math
import random

import torch
from torch.utils.checkpoint import checkpoint

import jaqsi_b200 as jq
from jaqsi_b200 import workloads as wl

# angles per wire and layer of each circuit family
_K = {"sweep": 3, "entangling": 3, "ring": 3, "crx": 1, "brick": 3, "noisy": 3}
_P, _GAMMA = 0.01, 0.005  # noise strengths of the noisy family


def listed():
    return [
        # one evaluation of a tiny circuit inside a host loop: latency alone
        _case("call_4q", "call", "sweep", 4, 2, "c128", out="expval"),
        # a small minibatch of the Hadamard + controlled-rotation ring (6 qubits, batch 10)
        _case("train_6q_b10", "train", "crx", 6, 4, "c128", batch=10),
        # a training step of a ten-qubit variational circuit, <Z_i> on every wire
        _case("train_10q", "train", "sweep", 10, 5, "c128"),
        # a minibatch of 64 samples through a 12-qubit classifier
        _case("train_12q_b64", "train", "ring", 12, 6, "c64", batch=64),
        # output distributions of a few parameter sets, 17 qubits
        _case("probs_17q_b8", "call", "entangling", 17, 8, "c64", out="probs", batch=8),
        # a final state in double precision, brickwork with CZ and RZZ entanglers
        _case("state_21q", "call", "brick", 21, 6, "c128", out="state"),
        # the large forward sweep: 24 qubits, 20 layers, ZZ chain
        _case("sweep_24q", "call", "sweep", 24, 20, "c64", out="expval", obs="zz"),
        # a gradient of 3000 angles on 20 qubits, ZZ chain
        _case("train_20q", "train", "entangling", 20, 50, "c64", obs="zz"),
        # a mid-size double precision gradient, three parameter sets
        _case("train_16q_b3", "train", "ring", 16, 9, "c128", batch=3, obs="zz"),
        # many circuits of 6 to 16 qubits and 10 to 40 layers at once
        _case("uneven_512", "uneven", "ring", 16, 40, "c64", batch=512),
        # noise-aware training of a small device, double precision minibatch
        _case("noisy_7q_b16", "train", "noisy", 7, 5, "c128", batch=16),
        # the largest: gradient through a noisy 12-qubit density matrix; eight
        # layers, since noise of this strength leaves a gradient of 1e-2 there
        # and of 6e-4 after twenty, of which float32 holds few digits
        _case("noisy_12q", "train", "noisy", 12, 8, "c64"),
    ]


def _case(name, kind, family, qubits, layers, dtype, out="expval", obs="z", batch=0):
    c = {"kind": kind, "family": family, "qubits": qubits, "layers": layers, "dtype": dtype, "out": out, "obs": obs,
         "batch": batch}
    return dict(c, name=name) if name else c


def _logint(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    dtype = rng.choice(["c64", "c128"])
    kind = rng.choice(["call", "call", "call", "train", "train", "train", "uneven", "noisy"])
    if kind == "uneven":
        return _case(None, "uneven", "ring", rng.randint(8, 16), rng.randint(8, 40), "c64", batch=_logint(rng, 16, 512))
    if kind == "noisy":
        n = rng.randint(2, 12)
        layers = rng.randint(1, 8 if dtype == "c64" else 20 if n < 11 else 4)
        batch = 0 if n > 8 else rng.choice([0, _logint(rng, 2, 24)])
        if rng.random() < 0.3:
            return _case(None, "call", "noisy", n, layers, dtype, out=rng.choice(["density", "probs", "expval"]), batch=batch)
        return _case(None, "train", "noisy", n, layers, dtype, batch=batch)
    family = rng.choice(["sweep", "entangling", "ring", "crx", "brick"])
    n = rng.randint(3, 24 if kind == "call" else 20)
    most = 1 << (23 if dtype == "c128" else 24)  # amplitudes of a call
    while 1 << n > most:
        n -= 1
    # (a Hadamard rounded to float32 loses norm at every use, so the crx
    # family stays shallow)
    layers = _logint(rng, 1, 8 if family == "crx" else 20 if kind == "call" or n > 16 else 50)
    batch = 0
    if n < 18 and rng.random() < 0.5:
        batch = _logint(rng, 2, max(2, min(256, (1 << 20) >> n)))
    if kind == "call":
        out = rng.choice(["expval", "expval", "probs", "state"])
        return _case(None, "call", family, n, layers, dtype, out=out, obs=rng.choice(["z", "zz"]), batch=batch)
    return _case(None, "train", family, n, layers, dtype, obs=rng.choice(["z", "zz"]), batch=batch)


# ---- the circuits, as a program writes them ---------------------------------
def _circuit(family, n, layers):
    if family == "sweep":
        return lambda a: wl.sweep_ansatz(n, layers, a)
    if family == "entangling":
        return lambda a: wl.strongly_entangling(n, layers, a)
    if family == "ring":
        return lambda a: wl.rot_ring(n, layers, a)
    if family == "noisy":
        return lambda a: wl.noisy_ansatz(n, layers, a, _P, _GAMMA)
    if family == "crx":
        def crx(a):
            for l in range(layers):
                for w in range(n):
                    jq.H(wires=w)
                for w in range(n):
                    jq.CRX(a[l, w, 0], wires=[w, (w + 1) % n])
        return crx

    def brick(a):
        for l in range(layers):
            for w in range(n):
                jq.RY(a[l, w, 0], wires=w)
                jq.RZ(a[l, w, 1], wires=w)
            for w in range(l % 2, n - 1, 2):
                if l % 3 == 2:
                    jq.CZ(wires=[w, w + 1])
                else:
                    jq.RZZ(a[l, w, 2], wires=[w, w + 1])
    return brick


def _obs(case):
    n = case["qubits"]
    if case["out"] != "expval":
        return []
    return wl.zz_chain(n) if case["obs"] == "zz" else wl.z_each(n)


def _shapes(case):
    """(qubits, depth) of every circuit of an uneven case: fixed by its sizes."""
    r = random.Random(1000 * case["qubits"] + case["layers"])
    lo = min(10, case["layers"])
    return [(r.randint(6, case["qubits"]), r.randint(lo, case["layers"])) for _ in range(case["batch"])]


def _params(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if case["dtype"] == "c64" else torch.float64
    if case["kind"] == "uneven":
        total = sum(3 * n * d for n, d in _shapes(case))
        return torch.rand(total, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    shape = (case["layers"], case["qubits"], _K[case["family"]])
    if case["batch"]:
        shape = (case["batch"],) + shape
    return torch.rand(shape, generator=g, device="cuda", dtype=dt) * (2 * math.pi)


_KEPT = {}  # what a program keeps between calls: its scripts and batch handles


def _kept(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _KEPT:
        if len(_KEPT) >= 32:
            _KEPT.pop(next(iter(_KEPT)))
        if case["kind"] == "uneven":
            items = []
            for n, d in _shapes(case):
                zero = [[[0.0] * 3] * n] * d
                with jq.recording() as tape:
                    for l in range(d):
                        for w in range(n):
                            jq.Rot(zero[l][w][0], zero[l][w][1], zero[l][w][2], wires=w)
                        for w in range(n):
                            jq.CX(wires=[w, (w + 1) % n])
                items.append((tape, n, [jq.PauliZ(0)]))
            _KEPT[key] = jq.BatchedGradients(items, dtype=torch.complex64)
        else:
            _KEPT[key] = jq.Script(_circuit(case["family"], case["qubits"], case["layers"]), case["qubits"])
    return _KEPT[key]


def prepare(case, seed):
    state = {"kind": case["kind"], "program": _kept(case), "params": _params(case, seed)}
    if case["kind"] != "uneven":
        state["params"].requires_grad_(case["kind"] == "train")
        state["call"] = {"type": case["out"], "obs": _obs(case),
                         "dtype": torch.complex64 if case["dtype"] == "c64" else torch.complex128,
                         "in_axes": (0,) if case["batch"] else None}
    return state


def run(state):
    program, params = state["program"], state["params"]
    if state["kind"] == "uneven":
        program.set_angles(params)
        return program.run()
    value = program.execute(args=(params,), **state["call"])
    if state["kind"] == "call":
        return value
    (grad,) = torch.autograd.grad(value.sum(), params)
    return value.detach(), grad


# ---- what a pass cannot do without -------------------------------------------
def _gates(case, n, layers):
    """(one-wire blocks, entanglers) of a circuit after fusing rotations of one wire."""
    if case["family"] == "brick":
        return n * layers, sum(len(range(l % 2, n - 1, 2)) for l in range(layers))
    return n * layers, n * layers


def work(case):
    """Bytes: parameters and results.  Flops: 14 per amplitude and one-wire
    complex 2x2 block, 30 per element of a density matrix and one-wire
    channel, entanglers that permute or phase counted at 0 or 6; a gradient
    undoes every block on two vectors and takes one inner product of it."""
    n, layers, batch = case["qubits"], case["layers"], max(1, case["batch"])
    real = 4 if case["dtype"] == "c64" else 8
    if case["kind"] == "uneven":
        shapes = _shapes(case)
        count = sum(3 * a * d for a, d in shapes)
        return {"bytes": 16 * count + 8 * len(shapes), "flops": sum((14 * 3 + 8) * a * d * 2.0**a for a, d in shapes)}
    angles = batch * layers * n * _K[case["family"]]
    size = {"expval": n if case["obs"] == "z" else n - 1, "probs": 2**n, "state": 2 * 2**n, "density": 2 * 4**n}[case["out"]]
    byts = real * (angles + batch * size)
    one, two = _gates(case, n, layers)
    if case["family"] == "noisy":
        flops = (one + 2 * two) * 30 * 4.0**n
    else:
        flops = (one * 14 + (two * 6 if case["family"] == "brick" else two * 7 if case["family"] == "crx" else 0)) * 2.0**n
    if case["kind"] == "train":
        byts += real * angles
        flops = flops * 3 + 8 * one * (4.0 if case["family"] == "noisy" else 2.0)**n
    return {"bytes": byts, "flops": flops * batch}


# ---- the same results from plain torch in 64 bits ------------------------------
def _rz(t):
    return torch.diag_embed(torch.stack([torch.exp(-0.5j * t), torch.exp(0.5j * t)], -1))


def _ry(t):
    c, s = torch.cos(t / 2), torch.sin(t / 2)
    return torch.stack([torch.stack([c, -s], -1), torch.stack([s, c], -1)], -2).to(torch.complex128)


def _rx(t):
    c, s = torch.cos(t / 2).to(torch.complex128), -1j * torch.sin(t / 2)
    return torch.stack([torch.stack([c, s], -1), torch.stack([s, c], -1)], -2)


def _one(x, u, w, bits):
    """u [B, 2, 2] on wire w of x [B, 2^bits]."""
    b = x.shape[0]
    v = x.reshape(b, 2**w, 2, 2 ** (bits - 1 - w))
    m = [[u[:, i, j].reshape(-1, 1, 1) for j in range(2)] for i in range(2)]
    a, c = v[:, :, 0], v[:, :, 1]
    return torch.stack([m[0][0] * a + m[0][1] * c, m[1][0] * a + m[1][1] * c], 2).reshape(b, -1)


def _two(x, u, w, v, bits):
    """u [B, 4, 4] on wires w < v (w the more significant)."""
    b = x.shape[0]
    y = x.reshape(b, 2**w, 2, 2 ** (v - 1 - w), 2, 2 ** (bits - 1 - v))
    s = [y[:, :, i >> 1, :, i & 1] for i in range(4)]
    r = [sum(u[:, i, j].reshape(-1, 1, 1, 1) * s[j] for j in range(4)) for i in range(4)]
    return torch.stack([torch.stack(r[:2], 3), torch.stack(r[2:], 3)], 2).reshape(b, -1)


def _cx(x, c, t, bits):
    b, lo, hi = x.shape[0], min(c, t), max(c, t)
    y = x.reshape(b, 2**lo, 2, 2 ** (hi - 1 - lo), 2, 2 ** (bits - 1 - hi))
    if c < t:
        return torch.stack([y[:, :, 0], y[:, :, 1].flip(3)], 2).reshape(b, -1)
    return torch.stack([y[:, :, :, :, 0], y[:, :, :, :, 1].flip(2)], 4).reshape(b, -1)


def _noise(device):
    """The noisy family's two channels in a row, as a map of (ket, bra) pairs."""
    c = torch.complex128
    eye, x = torch.eye(2, dtype=c), torch.tensor([[0, 1], [1, 0]], dtype=c)
    y, z = torch.tensor([[0, -1j], [1j, 0]], dtype=c), torch.diag(torch.tensor([1, -1], dtype=c))
    dep = [math.sqrt(1 - _P) * eye] + [math.sqrt(_P / 3) * m for m in (x, y, z)]
    amp = [torch.tensor([[1, 0], [0, math.sqrt(1 - _GAMMA)]], dtype=c), torch.tensor([[0, math.sqrt(_GAMMA)], [0, 0]], dtype=c)]
    both = [sum(torch.kron(k, k.conj()) for k in ks) for ks in (dep, amp)]
    return (both[1] @ both[0]).to(device)


def _layer(family, n, l, x, a):
    """Layer l of a family on x [B, 2^n] (noisy: [B, 4^n]) with angles a [B, n, k]."""
    if family == "noisy":
        ch = _noise(x.device)
        for w in range(n):
            s = None
            for k, f in enumerate((_rx, _ry, _rz)):
                u = f(a[:, w, k])
                m = ch @ torch.einsum("bij,bkl->bikjl", u, u.conj()).reshape(-1, 4, 4)
                s = m if s is None else m @ s
            x = _two(x, s, w, n + w, 2 * n)
        for w in range(n):
            v = (w + 1) % n
            x = _cx(_cx(x, w, v, 2 * n), n + w, n + v, 2 * n)
            for q in (w, v):
                x = _two(x, ch[None], q, n + q, 2 * n)
        return x
    if family == "crx":
        h = torch.tensor([[1, 1], [1, -1]], dtype=x.dtype, device=x.device)[None] / math.sqrt(2)
        for w in range(n):
            x = _one(x, h, w, n)
        for w in range(n):
            v, u = (w + 1) % n, _rx(a[:, w, 0])
            full = torch.diag_embed(torch.ones(u.shape[0], 4, dtype=u.dtype, device=u.device))
            at = (2, 3) if w < v else (1, 3)
            place = torch.zeros(4, 2, dtype=u.dtype, device=u.device)
            place[at[0], 0] = place[at[1], 1] = 1
            full = full - place @ place.T + place @ u @ place.T
            x = _two(x, full, min(w, v), max(w, v), n)
        return x
    for w in range(n):
        t = a[:, w]
        if family == "sweep":
            u = _rz(t[:, 2]) @ _ry(t[:, 1]) @ _rx(t[:, 0])
        elif family == "brick":
            u = _rz(t[:, 1]) @ _ry(t[:, 0])
        else:
            u = _rz(t[:, 2]) @ _ry(t[:, 1]) @ _rz(t[:, 0])
        x = _one(x, u, w, n)
    if family == "brick":
        for w in range(l % 2, n - 1, 2):
            if l % 3 == 2:
                u = torch.diag(torch.tensor([1, 1, 1, -1], dtype=x.dtype, device=x.device))[None]
            else:
                e = torch.exp(-0.5j * a[:, w, 2])
                u = torch.diag_embed(torch.stack([e, e.conj(), e.conj(), e], -1))
            x = _two(x, u, w, w + 1, n)
        return x
    r = (l % (n - 1)) + 1 if family == "entangling" else 1
    for w in range(n):
        x = _cx(x, w, (w + r) % n, n)
    return x


def _start(batch, bits):
    x = torch.zeros(batch, 2**bits, dtype=torch.complex128, device="cuda")
    x[:, 0] = 1
    return x


def _z_values(p, words, n):
    """Values of Z words (lists of wires) from probabilities p [B, 2^n]."""
    b, out = p.shape[0], []
    for ws in words:
        v = p
        for w in ws:
            y = v.reshape(b, 2**w, 2, -1)
            v = torch.stack([y[:, :, 0], -y[:, :, 1]], 2).reshape(b, -1)
        out.append(v.sum(1))
    return torch.stack(out, 1)


def _words(case):
    n = case["qubits"]
    return [[i, i + 1] for i in range(n - 1)] if case["obs"] == "zz" else [[i] for i in range(n)]


def exact(case, seed):
    p = _params(case, seed)
    if case["kind"] == "uneven":
        return _exact_uneven(case, p)
    a = p.detach().to(torch.float64)
    a = (a if case["batch"] else a[None]).requires_grad_(case["kind"] == "train")
    n, noisy = case["qubits"], case["family"] == "noisy"
    x = _start(a.shape[0], 2 * n if noisy else n)
    for l in range(case["layers"]):
        step = lambda y, t, l=l: _layer(case["family"], n, l, y, t)  # noqa: E731
        x = checkpoint(step, x, a[:, l], use_reentrant=False) if a.requires_grad else step(x, a[:, l])
    if noisy:
        x = x.reshape(-1, 2**n, 2**n)
        probs = torch.diagonal(x, dim1=1, dim2=2).real
    else:
        probs = x.abs().square() if not a.requires_grad else x.real.square() + x.imag.square()
    value = x if case["out"] in ("state", "density") else probs if case["out"] == "probs" else _z_values(probs, _words(case), n)
    if case["kind"] == "call":
        return value if case["batch"] else value[0]
    (grad,) = torch.autograd.grad(value.sum(), a)
    value = value.detach()
    return (value, grad) if case["batch"] else (value[0], grad[0])


def _exact_uneven(case, p):
    shapes, starts, at = _shapes(case), [], 0
    for n, d in shapes:
        starts.append(at)
        at += 3 * n * d
    values = torch.zeros(len(shapes), dtype=torch.float64, device="cuda")
    grads = torch.zeros_like(p)
    for n in sorted({s[0] for s in shapes}):
        # circuits of one size, deepest first: layer l runs those deeper than l
        mine = sorted((i for i, s in enumerate(shapes) if s[0] == n), key=lambda i: -shapes[i][1])
        depth = [shapes[i][1] for i in mine]
        a = torch.zeros(len(mine), depth[0], n, 3, dtype=torch.float64, device="cuda")
        for k, i in enumerate(mine):
            a[k, :depth[k]] = p[starts[i]:starts[i] + 3 * n * depth[k]].reshape(depth[k], n, 3)
        a.requires_grad_(True)
        x = _start(len(mine), n)
        for l in range(depth[0]):
            k = sum(d > l for d in depth)
            y = checkpoint(lambda y, t, l=l: _layer("ring", n, l, y, t), x[:k], a[:k, l], use_reentrant=False)
            x = torch.cat([y, x[k:]]) if k < len(mine) else y
        v = _z_values(x.real.square() + x.imag.square(), [[0]], n)[:, 0]
        (g,) = torch.autograd.grad(v.sum(), a)
        for k, i in enumerate(mine):
            values[i] = v[k].detach()
            grads[starts[i]:starts[i] + 3 * n * depth[k]] = g[k, :depth[k]].reshape(-1)
    return values, grads

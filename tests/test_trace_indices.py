"""What a call keeps and skips on the host: the index tensors of a cached trace
(usable by every later call, whatever was open around the first one, on any
stream), and the autograd Function (not inside torch.jit.trace and torch.func)."""
import pytest
import torch

import jaqsi_b200 as jq
from jaqsi_b200 import script as S
from jaqsi_b200 import simulation as sim

CPU = torch.device("cpu")


class _Lowered:
    def __init__(self, n):
        self.angles = [0.0] * n


def _trace(parts, cpos=(), cval=()):
    n = sum(len(p[1]) for p in parts) + len(cpos)
    return S._Trace(_Lowered(n), n, False, parts, list(cpos), list(cval))


ONE = [(0, [0, 1, 2], [0, 1, 2])]
SHARED = [(0, [0, 2], [1, 1]), (1, [1], [0])]


@pytest.mark.parametrize("parts,cpos,cval", [(ONE, (), ()), (SHARED, (), ()), (ONE, (3,), (0.5,))])
@pytest.mark.parametrize("batched", [False, True])
def test_first_call_in_inference_mode_then_a_gradient(parts, cpos, cval, batched):
    tr = _trace(parts, cpos, cval)
    args = (torch.rand(4, 3), torch.rand(3)) if batched else (torch.rand(3), torch.rand(3))
    how = (4, (0, None)) if batched else ()
    with torch.inference_mode():
        tr.angles(args, CPU, *how)
    args = tuple(a.clone().requires_grad_(True) for a in args)
    got = tr.angles(args, CPU, *how)
    got.sum().backward()
    want = torch.zeros(3, dtype=torch.float64)
    for _, _, idx in parts[:1]:
        for k in idx:
            want[k] += 1
    assert torch.equal(args[0].grad.double(), want.expand(args[0].shape))
    assert got.shape[-1] == tr.n_angles


def test_first_call_inside_a_torch_func_transform_keeps_plain_tensors():
    tr = _trace(SHARED, (3,), (0.5,))
    x = torch.rand(3)
    torch.func.grad(lambda y: tr.angles((y, y), CPU).sum())(x)
    kept = [t for k in (tr.cpos, tr.cval, *[q for p in tr.parts for q in p[1:]]) for t, _ in k.at.values()]
    assert len(kept) == 6 and not any(sim._functorch_wrapped(t) for t in kept)


@pytest.mark.gpu
def test_indices_outlive_a_dropped_trace_while_another_stream_reads_them():
    """A trace made on one stream and used on a second is dropped before the
    second has read its indices: their memory is not handed out again."""
    script = jq.Script(lambda p: jq.RY(p[0], wires=0) and None, n_qubits=1)
    p = torch.rand(1, device="cuda", dtype=torch.float64)
    obs = [jq.PauliZ(0)]
    read = []

    class Watch(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            if getattr(func, "__name__", "") == "index_select":
                read.append(args[2].data_ptr())
            return func(*args, **(kwargs or {}))

    script.execute("expval", obs, args=(p,))
    script.execute("expval", obs, args=(p,))  # replays the trace
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        torch.cuda._sleep(200_000_000)  # 0.1 s
        with Watch():
            script.execute("expval", obs, args=(p,))
    assert len(read) == 1
    script._jit_cache.clear()
    taken = [torch.empty(1, dtype=torch.long, device="cuda") for _ in range(64)]
    busy = not other.query()
    assert busy, "the second stream finished too early to tell"
    assert read[0] not in [t.data_ptr() for t in taken]
    torch.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("noisy", [False, True])
def test_traced_calls_run_the_circuit(noisy):
    """torch.jit.trace records the call as an autograd Function: the traced module
    runs it on other inputs."""

    def circuit(p):
        for w in range(2):
            jq.RY(p[w], wires=w)
            if noisy:
                jq.DepolarizingChannel(0.1, wires=w)

    script = jq.Script(circuit, n_qubits=2)
    obs = [jq.PauliZ(0), jq.PauliZ(1)]
    x = torch.tensor([0.3, 0.4], dtype=torch.float64, device="cuda")

    def call(p):
        return script.execute("expval", obs, args=(p,))

    want = call(x + 1)
    traced = torch.jit.trace(call, (x,), check_trace=False)
    assert torch.equal(traced(x + 1), want) and torch.equal(traced(x), call(x))


@pytest.mark.gpu
@pytest.mark.parametrize("noisy", [False, True])
def test_circuits_without_parameters_inside_torch_func(noisy):
    """Inside a transform buffers are wrappers: a circuit that takes nothing from it
    still runs."""

    def circuit(*p):
        jq.H(wires=0)
        jq.CX(wires=[0, 1])
        if noisy:
            jq.DepolarizingChannel(0.3, wires=1)

    script = jq.Script(circuit, n_qubits=2)
    obs = [jq.build_parity_observable([0, 1])]
    value = script.execute("expval", obs)
    x = torch.tensor([2.0, 3.0], dtype=torch.float64, device="cuda")

    def f(y):
        return (y * y * script.execute("expval", obs)).sum()

    assert torch.allclose(torch.func.grad(f)(x), 2 * x * value)
    assert torch.allclose(torch.func.jvp(f, (x,), (torch.ones_like(x),))[1], (2 * x * value).sum())
    assert torch.allclose(torch.func.vmap(lambda y: y * script.execute("expval", obs)[0])(x), x * value)

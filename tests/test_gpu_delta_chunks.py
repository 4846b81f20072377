"""The gated delta rule over long portions of heads with 128 rows, which go 64 tokens at a time on the tensor cores: edges of chunks, single
tokens, short and empty portions beside long ones, states carried over, a workspace that does not hold the chunks, values that are not finite."""
import pytest
import torch

from plain_vaderax import delta_rule, softplus, unit_vector
from test_gpu_vifelix import _batch, _ops, _run

pytestmark = pytest.mark.gpu
DEV, N = "cuda:0", 128
# Relative to the norm of the outputs: a sum of 128 products or decays, each with a rounding of 2^-24 of either sign, is off by sqrt(128) of
# them; half as much again for the exponentials of the gates.
TOL = 1.5 * 128 ** 0.5 * 2.0 ** -24


def _case(lens, H, G, p, seed):
    g = torch.Generator().manual_seed(seed)
    T = sum(lens)
    x, gates = torch.randn(T, 2 * G * N + H * p + 4, generator=g), 2 * torch.randn(T, 2 * H, generator=g)
    for t in range(3, T, 5):
        x[t, G * N:2 * G * N] = x[t - 2, G * N:2 * G * N]                # keys come again
    gates[T // 3::17, :H], gates[T // 4::23, :H] = 80.0, -80.0           # strengths of one and zero
    gates[T // 5::29, H:], gates[T // 2::13, H:] = 300.0, -80.0          # decays of zero and one
    return {"lens": lens, "H": H, "G": G, "p": p, "x": x, "gates": gates, "a_log": torch.randn(H, generator=g) - 1, "dt_bias": torch.randn(H, generator=g) - 2,
            "state": 0.1 * torch.randn(len(lens) + 1, H, p, N, generator=g)}


def _go(c, chunks=True):
    """Outputs [T, H, p] and states by request, from the kernels.  With `chunks` the workspace is the one that Runtime.delta_workspace gives; the
    memory behind what eight tokens at a time need of it shows whether 64 at a time ran."""
    lens, H, G, p, T, ops = c["lens"], c["H"], c["G"], c["p"], sum(c["lens"]), _ops()
    x, gates, state = c["x"].to(DEV), c["gates"].to(DEV), c["state"].to(DEV)
    eight = (T // 8 + len(lens) + 1) * H * 160
    floats = max(eight, (T // 64 + T // 256 + 1) * H * 8448 if chunks else 0)
    unit, coef, out = torch.full((T, 2 * G * N), float("nan"), device=DEV), torch.full((floats,), float("nan"), device=DEV), torch.zeros(T, H * p, device=DEV)
    slots = [len(lens) - r for r in range(len(lens))]
    _run(ops, lambda pl: pl.delta_rule(q=x[:, :G * N], k=x[:, G * N:2 * G * N], v=x[:, 2 * G * N:2 * G * N + H * p], write=gates[:, :H], forget=gates[:, H:],
                                          dt_bias=c["dt_bias"].to(DEV), a_log=c["a_log"].to(DEV), q_scale=N ** -0.5, unit_eps=1e-6, state=state, out=out,
                                          heads=H, n=N, p=p, qk_groups=G, unit=unit, coef=coef), _batch(lens, slots))
    assert torch.equal(state[0].cpu(), c["state"][0])                    # a slot of no request
    assert bool(torch.isfinite(coef[eight:]).any()) == (chunks and max(lens) >= 256)
    assert int(ops._lib("delta_rule").llme_delta_status()) == 0
    return out.view(T, H, p).cpu(), [state[s].cpu() for s in slots]


@pytest.mark.parametrize("lens,H,G,p", [([256], 1, 1, 32), ([319], 2, 1, 96), ([320], 3, 3, 32), ([321], 2, 2, 128), ([1, 600, 2, 509, 1], 4, 2, 64), ([1, 577], 6, 2, 32),
                                        ([63, 65, 64, 1100], 2, 1, 32), ([1500], 16, 8, 128)])
@pytest.mark.parametrize("chunks", [True, False])
def test_long_portions(lens, H, G, p, chunks):
    c = _case(lens, H, G, p, sum(lens) + p)
    y, states = _go(c, chunks)
    first = 0
    for r, L in enumerate(lens):
        s = slice(first, first + L)
        first += L
        heads = lambda x: x.reshape(L, G, N).double().repeat_interleave(H // G, 1)
        beta = torch.sigmoid(c["gates"][s, :H].double())
        keep = torch.exp(-torch.exp(c["a_log"].double()) * softplus(c["gates"][s, H:].double() + c["dt_bias"].double()))
        x = c["x"][s]
        want, S = delta_rule(unit_vector(heads(x[:, :G * N])) * N ** -0.5, unit_vector(heads(x[:, G * N:2 * G * N])), x[:, 2 * G * N:2 * G * N + H * p].reshape(L, H, p).double(),
                             beta, keep, c["state"][len(lens) - r].double().transpose(1, 2))
        assert float((y[s] - want).norm()) < TOL * float(want.norm()), r
        assert float((states[r].transpose(1, 2) - S).norm()) < TOL * float(S.norm()), r


@pytest.mark.parametrize("lens", [[250] + [1] * 10 + [600], [700, 3, 2], [256, 255, 257, 2, 500], [40] * 9 + [300] + [7] * 30 + [900, 5, 256], [200, 210, 190, 255, 254]])
def test_a_request_does_not_depend_on_its_neighbours(lens):
    """Outputs and states of every request are those of a step that it has to itself, bit for bit."""
    c = _case(lens, 4, 2, 64, sum(lens))
    y, states = _go(c)
    first = 0
    for r, L in enumerate(lens):
        s = slice(first, first + L)
        first += L
        own, kept = _go({**c, "lens": [L], "x": c["x"][s], "gates": c["gates"][s], "state": c["state"][[0, len(lens) - r]]})
        assert torch.equal(y[s], own) and torch.equal(states[r], kept[0]), (r, L)


def test_empty_portions_beside_long_ones():
    """They write nothing: outputs and states of the others are those of a step without them, and their own states stay."""
    c = _case([0, 600, 0, 700, 0], 2, 1, 32, 11)
    d = {**c, "lens": [600, 700], "state": c["state"][[0, 2, 4]]}        # (request r's state is slot len(lens) - r)
    (y, states), (want, kept) = _go(c), _go(d)
    assert torch.equal(y, want) and torch.equal(states[1], kept[0]) and torch.equal(states[3], kept[1])
    for r in (0, 2, 4):
        assert torch.equal(states[r], c["state"][5 - r])


def test_values_that_are_not_finite_reach_no_token_before_them():
    lens, H, G, p = [400, 300], 2, 1, 64
    c = _case(lens, H, G, p, 7)
    c["gates"][:, H:] = c["gates"][:, H:].clamp(max=2.0)                 # (nothing is forgotten at once)
    clean, _ = _go(c)
    c["x"][100, 2 * N + 5] = float("inf")                                # first request: one column of the first head
    c["x"][500, N + 3] = float("nan")                                    # the second one: a key of both heads
    c["x"][420, 7] = float("nan")                                        # and before it a query, which nothing keeps
    y, states = _go(c)
    bad = torch.zeros_like(y, dtype=torch.bool)
    bad[100:400, 0, 5] = bad[500:] = bad[420] = True
    assert bool((torch.isfinite(y) == ~bad).all())
    assert float((y[~bad] - clean[~bad]).norm()) < 2 * TOL * float(clean[~bad].norm())
    assert not bool(torch.isfinite(states[1]).any()) and bool(torch.isfinite(states[0][1]).all()) and not bool(torch.isfinite(states[0][0, 5]).any())

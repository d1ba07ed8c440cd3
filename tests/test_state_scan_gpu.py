"""The scan over matrix states (csrc/state_scan.cu) with one, two and four columns per thread, for each step of a token, against the
fp32 restatements of its callers on the CPU."""
import pytest
import torch

from sllm_b200.engine.batch import make_prefill_batch
from sllm_b200.ops import delta as D
from sllm_b200.ops import linear_state as S
from sllm_b200.ops.core import LinearWeight

pytestmark = pytest.mark.gpu
DEV = "cuda"
# heads, keys, values, columns per thread for four sequences: lanes per column 1, 4 and 8, values that no tile and no access divides
SIZES = [(8, 64, 70, 1), (15, 64, 70, 2), (16, 64, 72, 2), (24, 64, 70, 4), (40, 64, 72, 4), (36, 16, 130, 2), (40, 16, 130, 4), (6, 128, 128, 2),
         (10, 128, 128, 4), (9, 100, 50, 1)]


def _columns(heads, keys, values, sequences):
    """The rule of scan_columns: as few columns as keep the grid within the SMs."""
    lanes = 1
    while lanes * 16 < keys:
        lanes *= 2
    ctas = lambda c: heads * -(-values // (4 * (32 // lanes) * c)) * sequences
    return 1 if ctas(1) <= 148 else 2 if ctas(2) <= 148 else 4


def _batch(counts, device):
    b = make_prefill_batch([[0] * n for n in counts], torch.zeros((len(counts), 1), dtype=torch.int32, device=device), device)
    b.slots = torch.tensor([3, 0, 4, 1], dtype=torch.int32, device=device)
    return b


def _compare(run, state):
    """run(device, state) -> [T, *]; results and states of both devices agree to fp32 sums in another order."""
    want_state, got_state = state.clone(), state.to(DEV)
    want, got = run("cpu", want_state).double(), run(DEV, got_state).double().cpu()
    assert (got - want).norm() < 3e-5 * want.norm() and (got - want).abs().max() < 2e-4 * want.abs().max()
    assert (got_state.cpu() - want_state).norm() < 3e-5 * want_state.norm()
    assert torch.equal(got_state[2].cpu(), state[2])                   # a slot of nobody


COUNTS = [9, 1, 20, 8]


@pytest.mark.parametrize("heads,keys,values,columns", SIZES)
def test_plain_step(heads, keys, values, columns):
    assert _columns(heads, keys, values, len(COUNTS)) == columns
    g = torch.Generator().manual_seed(heads + values)
    col, at = {}, 0
    for n, w in (("q", heads * keys), ("k", heads * keys), ("v", heads * values), ("g", heads * values)):
        col[n], at = at, at + (w + 7) // 8 * 8
    spec = S.StateSpec(S.FIXED, heads, heads, keys, values, col, q_scale=keys ** -0.5)
    rate, proj = 0.5 + 0.5 * torch.rand(heads, generator=g), torch.randn(sum(COUNTS), at, generator=g)
    _compare(lambda dev, st: S.linear_state(proj.to(dev), spec, S.StateWeights(rate=rate.to(dev)), 1e-5, st, None, _batch(COUNTS, dev)),
             torch.randn(5, heads, keys, values, generator=g))


@pytest.mark.parametrize("heads,keys,values,columns", SIZES)
def test_gated_delta_step(heads, keys, values, columns):
    assert _columns(heads, keys, values, len(COUNTS)) == columns
    g = torch.Generator().manual_seed(heads + values)
    col, at = {}, 0
    for n, w in (("q", heads * keys), ("k", heads * keys), ("v", heads * values), ("g", heads * values), ("a", heads), ("b", heads)):
        col[n], at = at, at + w
        if n not in ("q", "k"):
            at = (at + 7) // 8 * 8
    spec = S.StateSpec(S.HEAD_DELTA, heads, heads, keys, values, col, q_scale=keys ** -0.5, taps=2)
    w = dict(bias=torch.randn(heads, generator=g) - 2, rate=torch.rand(heads, generator=g),
             conv_w=0.7 * torch.randn(2, 2 * heads * keys + heads * values, generator=g), norm=1 + 0.3 * torch.randn(values, generator=g))
    proj = torch.randn(sum(COUNTS), at, generator=g)

    def run(dev, st):
        ring = torch.zeros(5, 2, spec.channels, device=dev)
        return S.linear_state(proj.to(dev), spec, S.StateWeights(**{n: x.to(dev) for n, x in w.items()}), 1e-5, st, ring, _batch(COUNTS, dev))

    _compare(run, torch.randn(5, heads, keys, values, generator=g))


@pytest.mark.parametrize("heads,dim,columns", [(9, 50, 1), (30, 50, 2), (40, 50, 4), (6, 128, 2), (10, 128, 4)])
def test_removal_step(heads, dim, columns):
    assert _columns(heads, dim, dim, len(COUNTS)) == columns
    g = torch.Generator().manual_seed(heads + dim)
    rank, n = 16, heads * dim
    spec = D.DeltaSpec(heads, dim, rank)
    rnd = lambda *s: torch.randn(*s, generator=g)
    proj, w2, w0, ab, norm = rnd(sum(COUNTS), 5 * n + rank), rnd(n, rank) * 0.2, rnd(n), rnd(n), rnd(n)

    def run(dev, st):
        b = _batch(COUNTS, dev)
        return D.general_delta(proj.to(dev), spec, LinearWeight("dense", w2.to(dev)), w0.to(dev), ab.to(dev), norm.to(dev), 1e-5, st, b.row_off,
                               b.slots, False)

    _compare(run, 0.1 * rnd(5, heads, dim, dim))

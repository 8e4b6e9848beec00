"""Chunk preparation and walk of HGRN2, gated linear attention and the state-space recurrence (64 < dim <= 128) at the edges of
their chunks (16 and 32 tokens) and rings of slots, against the token-by-token restatement, with bars of the one-launch forms' tests."""
import pytest
import torch

from test_gpu_core_ops import gla_inputs, gla_want, ssd_inputs, ssd_want
from test_gpu_hybrid_ops import DEV, Batch, _hgrn2_inputs, _hgrn2_want, close, hops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,vdim", [(5, 128, 128), (2, 72, 8), (3, 96, 136)])
@pytest.mark.parametrize("lengths", [[33], [64, 1, 65, 16], [81] + [1, 2, 17] * 44])
def test_hgrn2_walk(hops, heads, dim, vdim, lengths):  # noqa: F811
    """One sequence, several, and more of them than a CTA looks through at once; states carried in every second one."""
    n, eps = len(lengths), 1e-5
    qfv, lower, bias, norm = _hgrn2_inputs(sum(lengths), heads, dim, vdim, torch.bfloat16, 51)
    before, starts = rnd(n, heads, dim, vdim, seed=52), [i % 2 for i in range(n)]
    slots, state = list(range(n))[::-1], before.to(DEV)
    batch = Batch(slots, starts, lengths)
    out = hops.hgrn2_prefill(*[t.to(DEV) for t in (qfv, lower, bias, norm)], state, batch, vdim, eps)
    row = 0
    for i, (slot, start, length) in enumerate(zip(slots, starts, lengths)):
        if i < 6 or 124 <= i:            # a CTA looks through 128 sequences at a time
            want, last = _hgrn2_want(qfv[row: row + length], lower, bias, norm, heads, dim, vdim,
                                     before[slot] if start else torch.zeros(heads, dim, vdim), eps, vdim)
            close(out[row: row + length], want, torch.bfloat16, f"length {length}", 2.0)
            close(state[slot], last, torch.float32, f"state after {length}", 4.0)
        row += length
    assert torch.isfinite(out).all() and torch.isfinite(state).all()


@pytest.mark.parametrize("segments", [None, (32, 9), (16, 17)])
@pytest.mark.parametrize("heads,dim,vdim,true", [(3, 128, 128, 100), (2, 80, 136, 136)])
def test_gla_walk(hops, heads, dim, vdim, true, segments):  # noqa: F811
    """A sequence full of NaN changes nothing in its neighbours."""
    lengths, slots, starts, eps = [257, 15, 48, 33], [0, 3, 2, 1], [0, 4, 0, 9], 1e-5
    qkv, z, gate = gla_inputs(heads, dim, vdim, sum(lengths), torch.bfloat16, seed=61)
    z[:, ::9] = -90.0
    qkv[:, 2 * heads * dim:].view(-1, heads, vdim)[..., true:] = 0
    qkv[257:272] = float("nan")
    bias, norm, before = rnd(heads * dim, seed=62) + 1.0, rnd(vdim, seed=63), rnd(4, heads, dim, vdim, seed=64)
    before[..., true:] = 0
    state, out = before.to(DEV), torch.empty(sum(lengths), heads * vdim, dtype=torch.bfloat16, device=DEV)
    hops.gla_prefill(qkv.to(DEV), z.to(DEV), bias.to(DEV), norm.to(DEV), gate.to(DEV), state, out, Batch(slots, starts, lengths), true,
                     dim ** -0.5, 8.0, eps, segments=segments)
    row = 0
    for slot, start, n in zip(slots, starts, lengths):
        if slot != 3:
            first = before[slot] if start else torch.zeros(heads, dim, vdim)
            want, last = gla_want(qkv[row: row + n], z[row: row + n], gate[row: row + n], bias, norm, heads, dim, vdim, true, dim ** -0.5,
                                  8.0, eps, first)
            close(out[row: row + n], want, torch.bfloat16, f"length {n}", 2.0)
            close(state[slot], last, torch.float32, f"state after {n}", 20.0)
        row += n


@pytest.mark.parametrize("heads,groups,dim,vdim", [(9, 1, 128, 64), (18, 2, 72, 48), (2, 2, 96, 112)])
@pytest.mark.parametrize("lengths,segments", [([33], None), ([64, 31, 65, 128, 1], None), ([401] + [1, 32, 40] * 90, None), ([257, 32, 200], (64, 5))])
def test_state_space_walk(hops, heads, groups, dim, vdim, lengths, segments):  # noqa: F811
    """Groups of more heads than a prep CTA takes, whole and part columns, more sequences than a CTA looks through at once."""
    n = len(lengths)
    xbc, step, dt_bias, a_log, skip = ssd_inputs(heads, groups, dim, vdim, sum(lengths), torch.bfloat16, seed=71)
    a_log = a_log - 3.0
    before, starts, slots = rnd(n, heads, dim, vdim, seed=72), [i % 2 for i in range(n)], list(range(n))[::-1]
    state = before.to(DEV)
    y = hops.ssd_prefill(xbc.to(DEV), step.to(DEV), *(t.to(DEV) for t in (dt_bias, a_log, skip)), state, groups, Batch(slots, starts, lengths),
                         segments=segments)
    row = 0
    for i, (slot, start, length) in enumerate(zip(slots, starts, lengths)):
        if i < 5 or 252 <= i:            # a CTA looks through 256 sequences at a time
            first = before[slot] if start else torch.zeros(heads, dim, vdim)
            want, last = ssd_want(xbc[row: row + length], step[row: row + length], dt_bias, a_log, skip, heads, groups, dim, vdim, first)
            close(y[row: row + length], want, torch.bfloat16, f"length {length}")
            close(state[slot], last, torch.float32, f"state after {length}", 20.0)
        row += length
    assert torch.isfinite(y).all() and torch.isfinite(state).all()


@pytest.mark.parametrize("lengths", [[300, 40], [60] * 6])
@pytest.mark.parametrize("kind", ["hgrn2", "gla", "ssd"])
def test_segments_to_spare(hops, kind, lengths):  # noqa: F811
    """More segments asked for than any sequence has: no CTA of the first pass has work, and what follows it still comes after the
    preparation.  Twice over the same memory, so that slots which were not written again would hold other values' fragments."""
    heads, dim, vdim, eps, n, total = 3, 128, 64, 1e-5, len(lengths), sum(lengths)
    batch, zero = Batch(list(range(n)), [0] * n, lengths), torch.zeros(heads, dim, vdim)
    for seed in (81, 91):
        state = torch.zeros(n, heads, dim, vdim, device=DEV)
        if kind == "hgrn2":
            qfv, lower, bias, norm = _hgrn2_inputs(total, heads, dim, vdim, torch.bfloat16, seed)
            out = hops.hgrn2_prefill(*[t.to(DEV) for t in (qfv, lower, bias, norm)], state, batch, vdim, eps, segments=(512, 2))

            def want(a, b):
                return _hgrn2_want(qfv[a:b], lower, bias, norm, heads, dim, vdim, zero, eps, vdim)
        elif kind == "gla":
            qkv, z, gate = gla_inputs(heads, dim, vdim, total, torch.bfloat16, seed=seed)
            bias, norm = rnd(heads * dim, seed=seed + 3) + 1.0, rnd(vdim, seed=seed + 4)
            out = torch.empty(total, heads * vdim, dtype=torch.bfloat16, device=DEV)
            hops.gla_prefill(*[t.to(DEV) for t in (qkv, z, bias, norm, gate)], state, out, batch, vdim, dim ** -0.5, 8.0, eps, segments=(512, 2))

            def want(a, b):
                return gla_want(qkv[a:b], z[a:b], gate[a:b], bias, norm, heads, dim, vdim, vdim, dim ** -0.5, 8.0, eps, zero)
        else:
            xbc, step, dt_bias, a_log, skip = ssd_inputs(heads, 1, dim, vdim, total, torch.bfloat16, seed=seed)
            a_log = a_log - 3.0
            out = hops.ssd_prefill(*[t.to(DEV) for t in (xbc, step, dt_bias, a_log, skip)], state, 1, batch, segments=(512, 2))

            def want(a, b):
                return ssd_want(xbc[a:b], step[a:b], dt_bias, a_log, skip, heads, 1, dim, vdim, zero)
        row = 0
        for i, length in enumerate(lengths):
            y, last = want(row, row + length)
            close(out[row: row + length], y, torch.bfloat16, f"length {length}", 2.0)
            close(state[i], last, torch.float32, f"state after {length}", 20.0)
            row += length


@pytest.mark.parametrize("kind,arg", [("hgrn2", 12), ("gla", 16), ("ssd", -3), ("gdn", 17)])
def test_batch_longer_than_named(hops, kind, arg, monkeypatch):  # noqa: F811
    """A call that names fewer tokens than its sequences hold: those within what was named are right, the others are left alone, and
    the flag that a kernel gave up is raised."""
    from b200attn import _lib, ops
    from helpers import gdn_inputs
    heads, dim, vdim, eps, lengths = 16, 128, 64, 1e-5, [70, 40, 200]
    n, total, batch = len(lengths), sum(lengths), Batch([0, 1, 2], [0] * 3, lengths)
    call = _lib.call

    def short(name, *args):
        args = list(args)
        args[arg] = 112                       # two sequences and a bit of the third
        return call(name, *args)

    def run():
        if kind == "gdn":
            out, state = ops.gdn_chunked_prefill_packed(*(t.to(DEV) for t in gdn_inputs(total, heads, torch.Generator().manual_seed(5))), batch.cu,
                                                        state_out=torch.full((n, heads, 128, 128), 7.0, device=DEV))
            return out, state
        state = torch.full((n, heads, dim, vdim), 7.0, device=DEV)
        if kind == "hgrn2":
            return hops.hgrn2_prefill(*[t.to(DEV) for t in _hgrn2_inputs(total, heads, dim, vdim, torch.bfloat16, 5)], state, batch, vdim, eps), state
        if kind == "gla":
            qkv, z, gate = (t.to(DEV) for t in gla_inputs(heads, dim, vdim, total, torch.bfloat16, seed=5))
            out = torch.empty(total, heads * vdim, dtype=torch.bfloat16, device=DEV)
            hops.gla_prefill(qkv, z, torch.ones(heads * dim, device=DEV), torch.ones(vdim, device=DEV), gate, state, out, batch, vdim, 0.1, 8.0, eps)
            return out, state
        return hops.ssd_prefill(*[t.to(DEV) for t in ssd_inputs(heads, 1, dim, vdim, total, torch.bfloat16, seed=5)], state, 1, batch), state

    want = run()
    torch.cuda.synchronize()
    assert _lib.load().b200_wait_timed_out() == 0
    monkeypatch.setattr(_lib, "call", short)
    got = run()
    torch.cuda.synchronize()
    assert _lib.load().b200_wait_timed_out() == 1
    assert torch.equal(got[0][:110], want[0][:110]) and torch.equal(got[1][:2], want[1][:2])
    assert torch.equal(got[1][2], torch.full_like(got[1][2], 7.0))

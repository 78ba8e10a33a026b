"""decay_chunk_kernel (recurrences with one decay per head, 128 tokens at a time) at the edges of its chunks, operand blocks and segments,
through the entry points that reach it, against the plain oracles.  Tolerances are those of the same entry points elsewhere: outputs are
rounded to bf16 (2^-9 of a value) and every factor has 16 bits."""
import math

import pytest
import torch

from mini_vllm_b200 import _cabi, ops
from oracle import vebonex as memory
from tests.step_helpers import gen, rel, run_steps
from tests.test_gpu_rasezen_ops import run_state_space, want_state_space

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def space_inputs(g, lens, heads, groups, n, vdim):
    mk = lambda *s: torch.randn(*s, generator=g).to(BF)
    return [{"x": mk(t, heads, vdim), "b": mk(t, groups, n), "c": mk(t, groups, n), "dt": mk(t, heads)} for t in lens]


@pytest.mark.parametrize("n,vdim", [(64, 64), (128, 64), (128, 128)])
@pytest.mark.parametrize("dt_bias,log_a", [(-4.0, 1.5), (-30.0, 0.0), (40.0, 3.0), (-1.0, -12.0)])
def test_state_space_edges(cuda, n, vdim, dt_bias, log_a):
    g, heads = gen(n + vdim), 4
    seqs = space_inputs(g, [1, 31, 127, 128, 129, 256, 300, 400], heads, 2, n, vdim)
    bias, a, d = torch.full((heads,), dt_bias), -torch.exp(log_a + torch.randn(heads, generator=g) * 0.1), torch.randn(heads, generator=g)
    for portions in ([[10 ** 6]], [[128, 33], [65, 1, 200]]):
        for x, s in zip(run_state_space(cuda, seqs, heads, bias, a, d, portions, BF), seqs):
            assert rel(x, want_state_space(s, bias, a, d)) < 6e-3


@pytest.mark.parametrize("n,vdim", [(64, 128), (128, 64)])
def test_state_space_segments(cuda, n, vdim):
    g, heads, lens = gen(n), 2, [1500, 71, 1, 1280]
    assert _cabi.load().mvb_state_space_scratch_bytes(0, sum(lens), len(lens), max(lens), heads, n, vdim, 1) > 0
    seqs = space_inputs(g, lens, heads, 1, n, vdim)
    bias, a, d = torch.full((heads,), -3.0), -torch.exp(torch.linspace(-9, 1, heads)), torch.ones(heads)
    for portions in ([[10 ** 6]], [[1100, 64, 300], [70, 1], [1], [1200]]):
        for x, s in zip(run_state_space(cuda, seqs, heads, bias, a, d, portions, BF), seqs):
            assert rel(x, want_state_space(s, bias, a, d)) < 6e-3


def test_a_neighbour_full_of_infinities(cuda):
    """What lies behind a sequence's last row in memory is read, and must not reach its outputs or its state."""
    g, heads = gen(1), 2
    seqs = space_inputs(g, [130, 70, 200, 5], heads, 1, 128, 64)
    for bad in (seqs[1], seqs[3]):
        for k in ("x", "b", "c"):
            bad[k][:] = math.inf
    bias, a, d = torch.zeros(heads), torch.tensor([-0.3, -2.0]), torch.ones(heads)
    got = run_state_space(cuda, seqs, heads, bias, a, d, [[10 ** 6], [10 ** 6], [77], [10 ** 6]], BF)
    for i in (0, 2):
        assert rel(got[i], want_state_space(seqs[i], bias, a, d)) < 6e-3


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128), (128, 64), (64, 192)])
@pytest.mark.parametrize("f_bias,swing", [(4.0, 1.0), (-8.0, 6.0), (0.0, 20.0)])
def test_matrix_memory_edges(cuda, dim, vdim, f_bias, swing):
    g, heads, cap, lens = gen(dim + vdim), 3, 15.0, [1, 31, 127, 128, 129, 300, 700, 256]
    mk = lambda *s: torch.randn(*s, generator=g).to(BF)
    seqs = [{"q": mk(t, heads, dim), "k": mk(t, heads, dim), "v": mk(t, heads, vdim), "gate": mk(t, heads * vdim),
             "f": (mk(t, heads) * swing).to(BF), "i": (mk(t, heads) * swing).to(BF)} for t in lens]
    fb, ib, nw = torch.full((heads,), f_bias), torch.full((heads,), -2.0), torch.rand(heads * vdim, generator=g) + 0.5
    capped = lambda x, bias: cap * torch.tanh((x.double() + bias.double()) / cap)
    want = []
    for s in seqs:
        x = {k: v.double() for k, v in s.items()}
        f, i = torch.nn.functional.logsigmoid(capped(s["f"], fb)), capped(s["i"], ib)
        o = torch.stack([memory.mlstm_memory(x["q"][:, h] * dim ** -0.5, x["k"][:, h], x["v"][:, h], i[:, h], f[:, h])[0] for h in range(heads)], dim=1)
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)
        want.append(o.flatten(1) * nw.double() * torch.sigmoid(x["gate"]))
    for portions in ([[10 ** 6]], [[128, 33], [65, 1, 200]]):
        n = len(seqs)
        states = tuple(torch.full(s, 3.0, device=cuda) for s in ((n + 2, heads, dim, vdim), (n + 2, heads, dim), (n + 2, heads)))
        got, status = [torch.full(w.shape, math.nan, dtype=torch.float64) for w in want], ops.new_status(cuda)

        def step(entries, cu, pos, slot):
            x = {k: torch.cat([seqs[i][k][lo:hi] for i, lo, hi in entries]).to(cuda) for k in seqs[0]}
            wide = torch.cat([x[k].flatten(1) for k in ("q", "k", "v")], dim=1)
            q, k, v = wide.split([heads * dim, heads * dim, heads * vdim], dim=1)
            out = torch.full((pos.numel(), heads, vdim), math.nan, dtype=BF, device=cuda)
            ops.mlstm(q.unflatten(1, (heads, dim)), k.unflatten(1, (heads, dim)), v.unflatten(1, (heads, vdim)), x["f"], fb.to(cuda), x["i"], ib.to(cuda),
                      cap, x["gate"], nw.to(cuda), out, states, slot, cu, pos, dim ** -0.5, 1e-6, status=status)
            at = 0
            for i, lo, hi in entries:
                got[i][lo:hi] = out[at:at + hi - lo].flatten(1).double().cpu()
                at += hi - lo
        run_steps(cuda, lens, portions, step)
        ops.check_status(status)
        for a, b in zip(got, want):
            assert rel(a, b) < 8e-3


def memory_step(cuda, lens, heads, dim, vdim, f_bias, i_bias, eps, states=None, slots=None, starts=None, seed=0, edit=None):
    """One ragged step of the matrix memory over new inputs, and what the plain oracle makes of it: outputs, and the state behind each
    sequence.  ``states`` are changed in place."""
    g, cap, nw = gen(seed), 15.0, torch.ones(heads * vdim)
    mk = lambda *s: torch.randn(*s, generator=g).to(BF)
    seqs = [{"q": mk(t, heads, dim), "k": mk(t, heads, dim), "v": mk(t, heads, vdim), "f": mk(t, heads), "i": mk(t, heads), "gate": mk(t, heads * vdim)}
            for t in lens]
    for s in seqs:
        if edit is not None:
            edit(s)
    fb, ib, starts = torch.full((heads,), f_bias), torch.full((heads,), i_bias), starts or [0] * len(lens)
    capped = lambda x, bias: cap * torch.tanh((x.double() + bias.double()) / cap)
    want, behind = [], []
    for j, s in enumerate(seqs):
        x = {k: v.double() for k, v in s.items()}
        f, i = torch.nn.functional.logsigmoid(capped(s["f"], fb)), capped(s["i"], ib)
        has = states is not None and starts[j] > 0 and 0 <= slots[j] < states[0].shape[0]
        front = lambda h: tuple(z[slots[j], h].double().cpu() for z in states) if has else None
        runs = [memory.mlstm_memory(x["q"][:, h] * dim ** -0.5, x["k"][:, h], x["v"][:, h], i[:, h], f[:, h], front(h)) for h in range(heads)]
        o = torch.stack([r[0] for r in runs], dim=1)
        want.append((o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)).flatten(1) * torch.sigmoid(x["gate"]))
        behind.append([torch.stack([r[1][m] for r in runs]) for m in range(3)])
    x = {k: torch.cat([s[k] for s in seqs]).to(cuda) for k in seqs[0]}
    q, k, v = torch.cat([x[n].flatten(1) for n in "qkv"], dim=1).split([heads * dim, heads * dim, heads * vdim], dim=1)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=cuda)
    pos = torch.cat([torch.arange(t) + at for t, at in zip(lens, starts)]).to(cuda)
    status, out = ops.new_status(cuda), torch.full((sum(lens), heads, vdim), math.nan, dtype=BF, device=cuda)
    ops.mlstm(q.unflatten(1, (heads, dim)), k.unflatten(1, (heads, dim)), v.unflatten(1, (heads, vdim)), x["f"], fb.to(cuda), x["i"], ib.to(cuda), cap,
              x["gate"], nw.to(cuda), out, states, None if slots is None else torch.tensor(slots, dtype=torch.int32, device=cuda), cu, pos, dim ** -0.5, eps,
              status=status)
    return list(out.flatten(1).double().cpu().split(lens)), want, behind, status


@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 64)])
def test_matrix_memory_goes_on(cuda, dim, vdim):
    """Prompts behind a state of random values, whose normaliser comes from memory while the first products already run: outputs (an eps that
    keeps their size visible), memory, normaliser and maximum against the oracle."""
    heads, lens, slots, g = 8, [330, 5, 128, 257, 364, 200], [3, 6, 0, 1, 7, 4], gen(3)
    states = tuple(x.to(cuda) for x in (torch.randn(9, heads, dim, vdim, generator=g), torch.randn(9, heads, dim, generator=g), torch.randn(9, heads, generator=g)))
    torch.empty(64 << 20, device=cuda).zero_()                       # the states are no longer in a cache
    got, want, behind, status = memory_step(cuda, lens, heads, dim, vdim, 4.0, -1.0, 0.5, states, slots, [7, 9, 0, 3, 1, 2])
    ops.check_status(status)
    for j, slot in enumerate(slots):
        assert rel(got[j], want[j]) < 8e-3
        # factors of 16 bits, fp32 sums of up to 364 terms
        assert all(rel(states[m][slot], behind[j][m]) < 3e-5 for m in range(3))


@pytest.mark.parametrize("dim,vdim", [(128, 64), (64, 128)])
def test_a_normaliser_that_all_but_cancels(cuda, dim, vdim):
    """Two opposite keys, the first a 20,000th weaker by the second's decay: what is left of n . q is a 20,000th of its terms.  Terms of
    16 bits leave it wrong by 7 %; fp32 weights (four roundings or exponentials of 2^-22 each, at random) by half a per cent."""
    def edit(s):
        s["f"][:], s["i"][:] = 0, 0
        k = s["k"][40].clone()
        s["k"][:] = 0
        s["k"][40], s["k"][41] = k * 1000, -k * 1000         # (n . q stays above the floor of its size)
        s["q"] *= 1000
    got, want, _, status = memory_step(cuda, [200, 230], 16, dim, vdim, 11.9, 0.0, 1e12, edit=edit)
    ops.check_status(status)
    errs = []
    for x, y in zip(got, want):
        x, y = (z.view(-1, 16, vdim)[41:128] for z in (x, y))
        errs.append((x * y).sum(-1) / (y * y).sum(-1) - 1)             # of the size of a head's row: the rounding to bf16 averages out
    err = float(torch.cat(errs).pow(2).mean().sqrt())
    assert err < 1e-2, err


def off(got, want):
    """2-norm of the difference over that of the result."""
    got, want = got.double().cpu(), want.double()
    return float((got - want).norm() / want.norm())


def space_step(cuda, lens, heads, groups, n, vdim, dt_bias, a, seed=0, state=None, slots=None, starts=None, edit=None, longest=None):
    """One ragged step of the state space over new inputs; the inputs, the outputs of each sequence and the status."""
    g, d = gen(seed), torch.ones(heads)
    seqs = space_inputs(g, lens, heads, groups, n, vdim)
    for s in seqs:
        if edit is not None:
            edit(s)
    bias = torch.full((heads,), dt_bias)
    x, b, c = torch.cat([torch.cat([s[k].flatten(1) for k in "xbc"], dim=1) for s in seqs]).to(cuda).split([heads * vdim, groups * n, groups * n], dim=1)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=cuda)
    pos = torch.cat([torch.arange(t) + at for t, at in zip(lens, starts or [0] * len(lens))]).to(cuda)
    status, out = ops.new_status(cuda), torch.full((sum(lens), heads, vdim), math.nan, dtype=BF, device=cuda)
    ops.state_space(x.unflatten(1, (heads, vdim)), b.unflatten(1, (groups, n)), c.unflatten(1, (groups, n)), torch.cat([s["dt"] for s in seqs]).to(cuda),
                    *(z.float().to(cuda) for z in (bias, a / math.log(2.0), d)), out, state,
                    None if slots is None else torch.tensor(slots, dtype=torch.int32, device=cuda), cu, pos, longest=max(lens) if longest is None else longest,
                    status=status)
    return seqs, list(out.cpu().split(lens)), status


def space_walk(s, bias, a, state=None):
    """The recurrence in 64 bits: outputs and the state behind it, from ``state`` [heads, n, vdim] or zero."""
    x, heads = {k: v.double() for k, v in s.items()}, s["x"].shape[1]
    b, c = (x[k].repeat_interleave(heads // x[k].shape[1], dim=1) for k in "bc")
    dt, ys = torch.nn.functional.softplus(x["dt"] + bias), []
    S = torch.zeros(heads, b.shape[2], x["x"].shape[2], dtype=torch.float64) if state is None else state.double().cpu()
    for t in range(dt.shape[0]):
        S = S * torch.exp(a.double() * dt[t])[:, None, None] + (dt[t][:, None] * b[t])[:, :, None] * x["x"][t][:, None, :]
        ys.append((S * c[t][:, :, None]).sum(1) + x["x"][t])
    return torch.stack(ys), S


@pytest.mark.parametrize("n,vdim", [(64, 64), (128, 128)])
def test_weak_decays_behind_strong_ones(cuda, n, vdim):
    """32 tokens that forget little at the end of chunks whose other tokens forget nearly everything: the sums of the decays are hundreds of
    times the differences that count.  The values enter in two bf16 parts, which leave up to 2^-17 of one, at random."""
    def edit(s):
        s["dt"][:96], s["dt"][96:128], s["x"][:96] = 6, -3, 0       # (no values where the steps are long: they would outweigh the others)
    state = torch.zeros(1, 4, n, vdim, device=cuda)
    a = -torch.tensor([1.0, 1.3, 0.7, 2.0])
    seqs, got, status = space_step(cuda, [128], 4, 2, n, vdim, 0.0, a, n, state, [0], edit=edit)
    ops.check_status(status)
    y, S = space_walk(seqs[0], 0.0, a)
    assert off(got[0], y) < 4e-3
    err = off(state[0], S)
    assert err < 2 ** -17, err


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128)])
def test_weak_forget_gates_behind_strong_ones(cuda, dim, vdim):
    """The same of the matrix memory (the first of two prompts); its gates' functions are those of CUDA, exact to a few ulps."""
    def edit(s):
        s["f"][:96], s["f"][96:128], s["i"] = -40, 8, s["i"] * 0.1
    states = tuple(torch.zeros(*s, device=cuda) for s in ((2, 3, dim, vdim), (2, 3, dim), (2, 3)))
    got, want, behind, status = memory_step(cuda, [128, 300], 3, dim, vdim, 0.0, 0.0, 0.5, states, [0, 1], edit=edit)
    ops.check_status(status)
    assert off(got[0], want[0]) < 4e-3
    errs = [off(x[0], y) for x, y in zip(states, behind[0])]
    assert max(errs[:2]) < 2 ** -18, errs


@pytest.mark.parametrize("dim,vdim", [(64, 128), (128, 64)])
def test_memory_keeps_fp32(cuda, dim, vdim):
    """The memory behind a prompt is as far from 64 bits as fp32 weights leave it (a handful of roundings and exponentials of 2^-23 each, at
    random): the values enter in three bf16 parts; two alone leave 2e-6."""
    states = tuple(torch.zeros(*s, device=cuda) for s in ((1, 3, dim, vdim), (1, 3, dim), (1, 3)))
    got, want, behind, status = memory_step(cuda, [520], 3, dim, vdim, 3.0, -1.0, 0.5, states, [0], seed=2)
    ops.check_status(status)
    errs = [off(x[0], y) for x, y in zip(states, behind[0])]
    assert off(got[0], want[0]) < 4e-3 and max(errs) < 8e-7, errs

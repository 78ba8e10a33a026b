"""Single tokens of many sequences through the gated delta rule: the kernel that streams states past persistent CTAs against the one that
takes a CTA per state, which smaller batches reach, on the same inputs."""
import pytest
import torch

from mini_vllm_b200 import ops
from tests.step_helpers import gen, rel

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("dtype", [BF, F32])
@pytest.mark.parametrize("heads,kv,dim,vdim,seqs", [(16, 16, 128, 128, 40), (4, 2, 128, 128, 257), (8, 8, 64, 64, 75), (6, 3, 100, 90, 100), (8, 8, 256, 64, 76),
                                                    (5, 1, 40, 127, 150), (6, 3, 100, 126, 100), (16, 4, 96, 128, 37), (3, 3, 250, 50, 201)])
def test_many_states(cuda, dtype, heads, kv, dim, vdim, seqs):
    g, small = gen(dim + vdim), 1
    mk = lambda *s: torch.randn(*s, generator=g).to(dtype).to(cuda)
    wide = mk(seqs, 2 * kv * dim + heads * vdim)
    q, k, v = wide.split([kv * dim, kv * dim, heads * vdim], dim=1)
    q, k, v = q.unflatten(1, (kv, dim)), k.unflatten(1, (kv, dim)), v.unflatten(1, (heads, vdim))
    a, b, gate = mk(seqs, heads * dim), mk(seqs, heads), mk(seqs, heads * vdim)
    exp_a, bias, norm = (torch.rand(*s, generator=g).to(cuda) for s in ((heads,), (heads * dim,), (vdim,)))
    state = torch.randn(seqs + 3, heads, dim, -(-vdim // 4) * 4, generator=g).to(cuda)
    state[..., vdim:] = 0
    slots = torch.randperm(seqs + 3, generator=g)[:seqs].to(torch.int32).to(cuda)
    pos = (torch.arange(seqs) % 5 * 7).to(cuda)                     # every fifth is a sequence's first token, over leftovers
    want_state, want = state.clone(), torch.empty(seqs, heads, vdim, dtype=dtype, device=cuda)
    got, status = torch.empty_like(want), ops.new_status(cuda)
    call = lambda lo, hi, out, st: ops.gated_delta(q[lo:hi], k[lo:hi], v[lo:hi], a[lo:hi], b[lo:hi], gate[lo:hi], exp_a, bias, norm, out[lo:hi], st,
                                                   slots[lo:hi], None, pos[lo:hi], dim ** -0.5, 1e-6, 1.3, status=status)
    for lo in range(0, seqs, small):
        call(lo, lo + small, want, want_state)
    call(0, seqs, got, state)
    ops.check_status(status)
    # the same fp32 sums of up to 256 terms, some in another order: a few times 2^-23 of the largest
    assert rel(got, want.cpu()) < (2 ** -8 if dtype == BF else 1e-5) and rel(state, want_state.cpu()) < 1e-6
    used = torch.zeros(seqs + 3, dtype=torch.bool)
    used[slots.long().cpu()] = True
    assert torch.equal(state[~used], want_state[~used])

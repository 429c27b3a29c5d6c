"""Truncated sampling (csrc/sampling.cu) over rows that begin at any place, with every combination of cuts."""
import pytest
import torch

import plain_ops

pytestmark = pytest.mark.gpu


# a vocabulary shorter than a 16-byte piece, odd ones (rows begin 0 to 3 floats off the boundary), one whose list of candidates overflows
# and one whose does not; without top-p and top-k (no list), with min-p above and below the k-th largest
@pytest.mark.parametrize("vocab", [1, 2, 3, 7, 1027, 4099, 65537])
@pytest.mark.parametrize("spread", [1.0, 6.0])
def test_a_row_off_the_boundary_is_cut_as_an_aligned_one(vocab, spread):
    from vapi_b200 import ops
    cases = [(1.0, 0, 1.0, 0.05), (1.0, 0, 1.0, 0.0), (0.8, 0, 0.9, 0.0), (0.8, 0, 0.9, 0.02), (1.2, 40, 1.0, 0.0), (1.2, 40, 1.0, 0.5),
             (1.2, 40, 0.8, 1e-6), (1.0, 5000, 0.999, 0.0), (1.0, 3, 1.0, 0.9)]
    R = len(cases)
    logits = (torch.randn(R, vocab, generator=torch.Generator().manual_seed(vocab)) * spread).cuda()
    f = lambda v, dt=torch.float32: torch.tensor(v, dtype=dt, device="cuda")
    inv_t, top_k = f([1.0 / c[0] for c in cases]), f([c[1] for c in cases], torch.int32)
    top_p, min_p = f([c[2] for c in cases]), f([c[3] for c in cases])
    seeds, draws = f(list(range(R)), torch.int64), f([7] * R, torch.int64)
    out, tau, cnt = ops.sample_truncated(logits, inv_t, top_k, top_p, min_p, seeds, draws, check=True)
    for r, (T, k, tp, mp) in enumerate(cases):
        alone = ops.sample_truncated(logits[r:r + 1].clone(), *(t[r:r + 1].contiguous() for t in (inv_t, top_k, top_p, min_p, seeds, draws)), check=True)
        assert [float(t) for t in alone] == [float(out[r]), float(tau[r]), float(cnt[r])], r
        ids, _, _ = plain_ops.truncated_survivors(logits[r].cpu().numpy(), 1.0 / T, k or None, tp, mp)
        assert int(cnt[r]) == len(ids) and int(out[r]) in set(ids.tolist()), (r, int(cnt[r]), len(ids))

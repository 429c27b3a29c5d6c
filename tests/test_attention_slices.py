"""How the keys of a decode step are cut when its sequences alone fill the device."""
import pytest
import torch


# (sequences, longest, slices) of 8 kv heads where the device holds 444 blocks: at most half of it (untouched by this rule), more than
# half, more than all; the edges at one and a half times 32 and 24 tiles of 64 keys, and the cap of four rounds of blocks
@pytest.mark.parametrize("seqs,longest,slices", [(27, 4096, 1), (28, 3008, 1), (28, 3072, 2), (55, 3072, 2), (56, 2240, 1), (56, 2304, 2), (64, 4096, 3),
                                                 (64, 1, 1), (64, 32768, 4), (300, 32768, 1)])
def test_a_full_step_is_only_cut_where_a_sequence_could_be_long(monkeypatch, seqs, longest, slices):
    from vapi_b200 import ops
    monkeypatch.setattr(ops, "_decode_limits", (444, 8))
    assert ops.attention_splits(seqs, 1, longest, 32, 8, True) == slices


@pytest.mark.gpu
@pytest.mark.parametrize("rounds", [0.5, 1.0])
@pytest.mark.parametrize("longest", [2200, 4097])
def test_full_steps_on_both_sides_of_the_rule(rounds, longest):
    from vapi_b200 import ops
    from test_kernels_gpu import _attention_case
    seqs = int(rounds * ops.decode_attention_limits()[0]) // 4 + 1
    lens = [(1, 1 + (37 * i) % 130) for i in range(seqs - 2)] + [(1, longest), (1, longest - 64)]
    _attention_case(ops, torch.bfloat16, 16, 4, 64, 64, lens, planted=True)

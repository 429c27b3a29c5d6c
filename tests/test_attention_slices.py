"""How the keys of a decode step are cut when its sequences alone fill the device."""
import pytest
import torch


# (sequences, longest, slices) of 8 kv heads where the device holds 444 blocks: more than half of it and all of it stay whole at any configured
# context (short sequences lose by every slice, and a captured step does not know their lengths); more than all: the edge at one and a half
# times 24 tiles of 64 keys, and the cap of four rounds of blocks
@pytest.mark.parametrize("seqs,longest,slices", [(27, 4096, 1), (28, 3008, 1), (28, 3072, 1), (28, 8192, 1), (32, 8192, 1), (32, 128000, 1), (55, 3072, 1),
                                                 (55, 32768, 1), (56, 2240, 1), (56, 2304, 2), (64, 2049, 1), (64, 4096, 3), (64, 8192, 4), (64, 1, 1),
                                                 (64, 32768, 4), (128, 8192, 2), (300, 32768, 1)])
def test_a_full_step_is_only_cut_where_a_sequence_could_be_long(monkeypatch, seqs, longest, slices):
    from vapi_b200 import ops
    monkeypatch.setattr(ops, "_decode_limits", (444, 8))
    assert ops.attention_splits(seqs, 1, longest, 32, 8, True) == slices


def test_the_captured_step_of_a_default_server_keeps_short_chats_whole(monkeypatch):
    """The bucket of 32 requests as the runner plans it: from the configured context, not from the sequences."""
    from vapi_b200 import ops
    from vapi_b200.config.runtime import ModelSection
    from vapi_b200.parts.attention import GQAttention
    monkeypatch.setattr(ops, "_decode_limits", (444, 8))
    part = GQAttention.__new__(GQAttention)
    part.nh, part.nkv, part.d, part.window, part.general = 32, 8, 64, 0, False
    assert part.decode_splits(32, ModelSection().max_context, 64, torch.bfloat16) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("rounds", [0.5, 1.0])
@pytest.mark.parametrize("longest", [2200, 4097])
def test_full_steps_on_both_sides_of_the_rule(rounds, longest):
    from vapi_b200 import ops
    from test_kernels_gpu import _attention_case
    seqs = int(rounds * ops.decode_attention_limits()[0]) // 4 + 1
    lens = [(1, 1 + (37 * i) % 130) for i in range(seqs - 2)] + [(1, longest), (1, longest - 64)]
    _attention_case(ops, torch.bfloat16, 16, 4, 64, 64, lens, planted=True)

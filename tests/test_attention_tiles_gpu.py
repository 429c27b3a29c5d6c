"""The list of row tiles that the tcgen05 attention walks in steps of many sequences."""
import pytest
import torch

from test_kernels_gpu import _attention_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vapi_b200 import ops as o
    o.strict_fp32()
    return o


# portions first, last and between decode tokens; more than 32 and more than 64 sequences; portions at the edges of a tile of 128 rows;
# sequences below the kernel's least length between those above it
@pytest.mark.parametrize("lens", [[(70, 70)] + [(1, 5 + 7 * i) for i in range(40)],
                                  [(1, 9 + i) for i in range(33)] + [(64, 200), (1, 70), (33, 33)],
                                  [(32, 32)] * 3 + [(31, 40), (128, 128), (1, 1)] + [(2, 60)] * 30 + [(129, 300), (65, 65)],
                                  [(1, 3)] * 66 + [(257, 260)]])
@pytest.mark.parametrize("nh,nkv", [(8, 2), (3, 1)])
def test_portions_among_many_sequences(ops, lens, nh, nkv):
    _attention_case(ops, torch.bfloat16, nh, nkv, 64, 64, lens, splits=1)

"""GPU: arguments that the Python calls refuse (csrc/py_attention.cpp), with tensors that are otherwise right."""
import pytest
import torch

from dadgpt_b200 import _lib
from dadgpt_b200 import attention as dad

pytestmark = pytest.mark.gpu


def test_an_empty_mask_is_refused(cuda):
    """A mask tensor without elements is no mask, not a request to draw one."""
    x = torch.zeros(2, 8, 64, dtype=torch.bfloat16, device=cuda)
    lse = torch.zeros(2, 8, device=cuda)
    ws = torch.empty(dad.flash_backward_bf16_workspace_bytes(2, 8, 64), dtype=torch.uint8, device=cuda)
    empty = torch.empty(0, dtype=torch.int32, device=cuda)
    with pytest.raises(_lib.DadAttnError) as e:
        dad.gpu_flash_attention_forward_bf16(x, lse, x, x, x, 2, 8, 64, 0.125, rate=0.1, mask_bits=empty)
    assert e.value.code == -1
    with pytest.raises(_lib.DadAttnError) as e:
        dad.gpu_flash_attention_backward_bf16(x, x, x, ws, x, x, lse, x, x, x, 2, 8, 64, 0.125, rate=0.1,
                                              mask_bits=empty)
    assert e.value.code == -1


def test_sizes_beyond_32_bits_are_refused(cuda):
    """They would be right in their lower 32 bits."""
    x = torch.zeros(2, 8, 64, device=cuda)
    lse = torch.zeros(2, 8, device=cuda)
    for sizes in ((2 + 2**32, 8, 64), (2, 8 + 2**32, 64), (2, 8, 64 - 2**32)):
        with pytest.raises(ValueError):
            dad.gpu_flash_attention_forward(x, lse, x, x, x, *sizes, 0.125)
    for pos in (2**32, 2**32 + 3, -2**32):
        with pytest.raises(IndexError):
            dad.decode_attention_f32(x[:, 0].reshape(-1), *(x[:, 0].reshape(-1) for _ in range(3)), x, x, pos, 0.125)

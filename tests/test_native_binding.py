"""The native argument checks behind dadgpt_b200.attention (csrc/py_attention.cpp), on the CPU."""
import pytest
import torch

from dadgpt_b200 import _lib
from dadgpt_b200 import attention as dad


@pytest.mark.parametrize("call", ["forward", "decode", "mask"])
def test_cpu_tensors_are_refused(call):
    x, lse = torch.zeros(2, 8, 64), torch.zeros(2, 8)
    with pytest.raises(ValueError, match="CUDA tensor"):
        if call == "forward":
            dad.gpu_flash_attention_forward(x, lse, x, x, x, 2, 8, 64, 0.125)
        elif call == "decode":
            dad.decode_attention_f32(x[0], x[0], x[0], x[0], x, x, 0, 0.125)
        else:
            dad.dropout_mask_bits(2, 8, 0.1, 1, out=torch.zeros(4, dtype=torch.int32))


def test_errors_of_the_library_carry_its_code():
    with pytest.raises(TypeError):
        _lib.native().fwd_f32()
    assert issubclass(_lib.DadAttnError, RuntimeError)

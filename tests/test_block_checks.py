"""What a block as one autograd node checks of its operands, as the operators do (CPU: nothing is launched)."""
import pytest
import torch

from brain_b200.ops import blocks


def _param(main_grad, w=None):
    p = torch.nn.Parameter(torch.zeros(24, 16, dtype=torch.bfloat16) if w is None else w)
    p.main_grad = main_grad
    return p


@pytest.mark.parametrize("main_grad", [torch.zeros(24, 16, dtype=torch.bfloat16), torch.zeros(16, 24), torch.zeros(16, 24).t(),
                                       torch.zeros(24, 32)[:, ::2]], ids=["type", "shape", "columns", "stride"])
def test_gradients_that_the_kernels_cannot_add_to_are_refused(main_grad):
    p = _param(main_grad)
    x, dy = torch.zeros(8, 16, dtype=torch.bfloat16), torch.zeros(8, 24, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):
        blocks._project_back(dy, x, p, p, None, 8, None)


def test_operands_of_a_projection_are_checked():
    x = torch.zeros(8, 16, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):
        blocks._project(x, torch.zeros(16, 24, dtype=torch.bfloat16).t(), None, 8, None)       # columns, not rows
    with pytest.raises(AssertionError):
        blocks._project(x, torch.zeros(24, 32, dtype=torch.bfloat16), None, 8, None)           # another inner size

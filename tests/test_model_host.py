"""Host-side logic of the runtime that needs no GPU."""
import types

import pytest

from llm_decode_kernels_b200.model import Model


@pytest.mark.parametrize("prefilled,gemm,attention,persistent,ctrl,want", [
    (False, 1, 0, False, 0, 0),      # another model's prompt: not this one's business
    (True, 1, 0, False, 0, 5), (True, 1, 0, True, 0, 5), (True, 0, 0, True, 0, 0),
    (True, 1, 1, False, 0, 1), (True, 1, 0, True, 4, 4)])
def test_step_error_covers_the_prompt_kernels(prefilled, gemm, attention, persistent, ctrl, want):
    K = types.SimpleNamespace(gemm_status=lambda: gemm, paged_attention_status=lambda: attention)
    m = types.SimpleNamespace(K=K, comm=None, persistent=persistent, _step_static={"ctrl": [0, ctrl]}, _prefilled=prefilled)
    assert Model.step_error(m) == want

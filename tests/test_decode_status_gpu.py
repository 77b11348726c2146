"""A kernel that gave up on a wait in a decode step: the step's tokens are not handed out.  The word that such a kernel writes is
written by the host here."""
from __future__ import annotations

import pytest
import torch

from tiny_models import TINY, random_tokens, tiny_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("logprobs", [0, 2])              # captured and pipelined, and step by step
def test_no_token_after_a_wait_that_ran_out(dtype, logprobs):
    from mrun_b200.engine.engine import Engine
    from mrun_b200.kernels import ops
    t = TINY["E"]
    engine = Engine.from_config(tiny_config("E"), t["seed"], dtype=dtype, std=t["std"], num_pages=64, max_requests=4)
    device = engine.executor.device
    word = ops.status_word(device, "gemm_f32_tc", {5: "the sums"})
    seen = []

    def on_token(i, token):
        seen.append(token)
        if len(seen) == 4:
            word.fill_(5)
    prompt = random_tokens(t["config"]["vocab_size"], 9, 3)
    with pytest.raises(ops.KernelError, match="gemm_f32_tc: .* waited longer"):
        engine.generate([prompt], max_tokens=40, ignore_eos=True, on_token=on_token, logprobs=logprobs)
    assert len(seen) <= 5                                 # a step that was in flight before has its token
    assert int(word.item()) == 0
    assert len(engine.generate([prompt], max_tokens=6, ignore_eos=True)[0].tokens) == 6

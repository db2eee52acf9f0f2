"""The smoke entry point: its check of generated tokens (CPU) and the whole pass with several seeds (GPU)."""
import sys
from pathlib import Path

import pytest
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import __graft_entry__ as entry                                     # noqa: E402
from openvino_b200.models import llama                              # noqa: E402
from openvino_b200.models.llm_config import TINY_LLAMA as CFG       # noqa: E402


def _case(seed):
    state = llama.effective_state(CFG, llama.random_float_state(CFG, seed=seed), torch.bfloat16)
    prompt = torch.randint(0, CFG.vocab_size, (7,), generator=torch.Generator().manual_seed(seed)).tolist()
    return state, prompt, llama.reference_generate(CFG, state, prompt, 6)


def test_reference_tokens_pass_and_near_ties_do_not_decide():
    state, prompt, want = _case(0)
    entry.check_tokens(CFG, state, prompt, want)
    # a path that leaves the reference's at a margin below the error is as good, whatever comes after it
    row = llama.reference_logits(CFG, state, torch.tensor(prompt + want[:3]))[-1]
    tie = dict(state)
    tie["lm_head"] = state["lm_head"].clone()
    other = (want[3] + 1) % CFG.vocab_size
    tie["lm_head"][other] = tie["lm_head"][want[3]] * (1 - 1e-4)
    assert int(row.argmax()) == want[3]
    path = want[:3] + [other]
    for _ in range(2):
        path.append(int(llama.reference_logits(CFG, tie, torch.tensor(prompt + path))[-1].argmax()))
    entry.check_tokens(CFG, tie, prompt, path)


@pytest.mark.parametrize("at", [0, 3, 5])
def test_wrong_tokens_fail(at):
    state, prompt, want = _case(1)
    row = llama.reference_logits(CFG, state, torch.tensor(prompt + want[:at]))[-1]
    wrong = list(want)
    wrong[at] = int(row.argsort(descending=True)[8])
    with pytest.raises(RuntimeError, match="token %d is" % at):
        entry.check_tokens(CFG, state, prompt, wrong)


def test_scales_as_the_device_holds_them():
    cfg = CFG.with_(weight_format="int4")
    w = llama.random_float_state(cfg, seed=2)
    ir, dev = llama.effective_state(cfg, w), llama.effective_state(cfg, w, torch.bfloat16)
    key = "layers.0.q_proj"
    assert not torch.equal(ir[key], dev[key]) and (ir[key] - dev[key]).norm() < 2.0 ** -8 * ir[key].norm()
    assert torch.equal(ir["embed_tokens"], dev["embed_tokens"])


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(6))
def test_smoke(seed):
    entry.smoke(seed)

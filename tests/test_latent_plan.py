"""Which form a step's latent attention takes (no GPU: the plan is made on the host)."""
import pytest
import torch

from llmx_b200.parts.base import Precision, StepShape
from llmx_b200.parts.latent_attention import LatentAttention


def _wide(heads, counts, histories, room=0):
    part = LatentAttention(64, heads, 128, 64, 128, None, 512, 0.1, 1e4, 64, 1e-6)
    part.precision, part._sms, part.w_uk = Precision.of("bfloat16"), 148, torch.empty(0, dtype=torch.bfloat16)
    plan = part.plan_step(StepShape(counts, None if room else histories, room=room))
    return None if plan.wide is None else plan


@pytest.mark.parametrize("heads,rows,history,made", [
    (16, 32, 0, True), (16, 31, 0, False), (16, 32, 1000, True), (16, 32, 2000, False), (16, 40, 2000, True), (16, 32, 4000, False), (16, 40, 4000, False),
    (16, 48, 4000, True), (16, 64, 8000, True), (16, 96, 12000, False), (16, 128, 12000, True), (32, 32, 4000, True), (32, 48, 5000, False), (32, 64, 5000, True),
    (32, 48, 6000, False), (32, 128, 16000, True)])
def test_few_rows_after_many_keys_take_the_form_that_is_faster_for_them(heads, rows, history, made):
    """Where the form that makes keys and values was measured slower than the general one (the table in parts/latent_attention.py), it
    is not taken."""
    assert (_wide(heads, [rows], [history]) is not None) == made


def test_several_requests_count_together():
    """Requests of few rows add up while their heads fit one group; a request beside them that brings one row stays with the general
    form, and every row belongs to one of the two.  In several groups every one walks all keys again."""
    plan = _wide(16, [32, 1, 32], [4000, 4000, 4000])
    assert plan is not None and plan.wide[1] == 2 and sum(r[1] for r in plan.runs) == 1
    assert _wide(16, [32, 1], [4000, 9]) is None
    assert _wide(16, [33] * 4, [2000] * 4) is not None and _wide(16, [33] * 4, None, room=2048) is not None
    assert _wide(16, [32] * 2, [8000] * 2) is None and _wide(16, [32] * 8, [4000] * 8) is None

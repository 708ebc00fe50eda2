"""How a mixer of several branches calls their cores, without a GPU: the cores record what they are called with."""
from types import SimpleNamespace

import pytest
import torch

from mini_llm_b200.parts.attention import DistanceBiasAttention
from mini_llm_b200.parts.projected import ParallelMixer
from mini_llm_b200.parts.recurrent import GatedLinearRecurrence


class Attention(DistanceBiasAttention):
    in_width = core_width = 4

    def __init__(self):
        pass


class Recurrence(GatedLinearRecurrence):
    in_width = core_width = 2

    def __init__(self):
        pass


def _run(first, second):
    mixer = ParallelMixer.__new__(ParallelMixer)
    mixer.branches, mixer.scales = [first, second], [0.5, 2.0]
    mixer.in_weight, mixer.out_weight = torch.zeros(6, 8), torch.zeros(8, 6)
    mixer.rt = SimpleNamespace(act_dtype=torch.float32, ops=SimpleNamespace(linear=lambda *a, **k: None))
    ctx = SimpleNamespace(ws=SimpleNamespace(buf=lambda name, rows, cols, dtype: torch.zeros(rows, cols, dtype=dtype)))
    mixer.forward(torch.zeros(3, 8), ctx, None, torch.zeros(3, 8))


def test_cores_that_are_replaced_are_called_as_before():
    seen = []

    class Mine(Attention):
        def core(self, proj, ctx, cache, out, out_scale=1.0):
            seen.append(("attention", proj.shape[1], out.shape[1], out_scale))

    class Other(Recurrence):
        def core(self, proj, ctx, cache, out, *, out_scale=1.0):
            seen.append(("recurrence", proj.shape[1], out.shape[1], out_scale))

    _run(Mine(), Other())
    assert seen == [("attention", 4, 4, 0.5), ("recurrence", 2, 2, 2.0)]


@pytest.mark.parametrize("marked", [True, False])
def test_the_second_core_goes_as_the_first_ones_company(marked):
    seen = []

    class Mine(Attention):
        def core(self, proj, ctx, cache, out, out_scale=1.0, company=None):
            seen.append(("attention", out_scale, company is not None))
            if company is not None:
                company()

        core.takes_company = True

    class Other(Recurrence):
        def core(self, proj, ctx, cache, out, out_scale=1.0, beside=False):
            seen.append(("recurrence", out_scale, beside))

        if marked:
            core.goes_beside = True

    _run(Mine(), Other())
    assert seen == [("attention", 0.5, marked), ("recurrence", 2.0, marked)]
    assert DistanceBiasAttention.core.takes_company and GatedLinearRecurrence.core.goes_beside

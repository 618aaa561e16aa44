"""Plans of launches ask the device how many SMs it has."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "koboldcpp_b200" / "csrc"


def test_no_plan_has_the_number_of_sms_written_out():
    found = []
    for path in sorted(CSRC.glob("*.c*")) + sorted(CSRC.glob("*.h")):
        for number, line in enumerate(path.read_text().splitlines(), 1):
            code = line.split("//")[0]
            if re.search(r"\b148\b", code) and "race" not in code.lower():  # (a developer's timeline has room for so many CTAs)
                found.append((path.name, number, code.strip()))
    # the one place that asks the device, when there is none
    assert [f[0] for f in found] == ["b200_common.cuh"], found


@pytest.mark.gpu
def test_launches_of_a_prompt_whose_mask_is_read_once():
    """The statistics count the launch that reads a prompt's mask ahead: one a layer where the cache has 12 tiles of 64 cells (two query heads a kv-head)."""
    from koboldcpp_b200.lib import F16
    from koboldcpp_b200.llama import SHAPES, LlamaModel
    m = LlamaModel(SHAPES["test-dense"], 2048, F16)
    try:
        m.init_random(3)
        m.finalize(64)
        m.decode(list(range(64)), 0)
        short = m.stats()["n_kernels"]
        m.decode(list(range(64)), 1400)
        assert m.stats()["n_kernels"] - short == SHAPES["test-dense"].n_layer
    finally:
        m.close()

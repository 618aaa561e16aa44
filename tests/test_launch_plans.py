"""Plans of launches ask the device how many SMs it has."""
import re
from pathlib import Path

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

"""The status word of a step is shared by all kernels with bounded waits: a code says which kernel gave up and where."""
from __future__ import annotations

import re

from nncpu_b200.kernels.library import CSRC


def test_every_code_has_one_meaning():
    seen = {}
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for body in re.findall(r"enum \w*Status : int \{([^}]*)\}", text):
            for name, code in re.findall(r"(\w+) = (\d+)", body):
                if int(code):
                    assert int(code) not in seen, f"{path.name}: {name} = {code} is also {seen[int(code)]}"
                    seen[int(code)] = f"{path.name}: {name}"
        assert not re.search(r"atomicExch\([^;]*status, \d", text), f"{path.name}: a code without a name"
    assert len(seen) >= 16

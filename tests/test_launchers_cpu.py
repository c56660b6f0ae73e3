"""What the launchers keep between calls, read from their sources: a kernel's limit of dynamic shared memory belongs to a device, so no
launcher may remember for the whole process that it was raised (a model on the process's second device would fail at its first launch)."""
import pathlib
import re

import arle_b200

CSRC = pathlib.Path(arle_b200.__file__).parent / "csrc"


def test_no_launcher_remembers_a_device_setting_per_process():
    sources = sorted(CSRC.glob("*.cu"))
    assert sources
    for f in sources:
        text = f.read_text()
        assert not re.search(r"static\s+bool\s+\w+\s*(\[\w*\])?\s*[={;]", text), f.name
        for flag in re.findall(r"static\s+(?:std::)?(?:atomic<bool>|once_flag)\s+\w+", text):
            raise AssertionError(f"{f.name}: {flag}")


def test_the_limit_is_kept_per_device():
    text = (CSRC / "common.cuh").read_text()
    body = text[text.index("class SharedLimit"):]
    assert "cudaGetDevice(&dev)" in body[: body.index("};")]

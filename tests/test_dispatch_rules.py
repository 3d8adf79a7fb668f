"""The rules that choose a launch's shape (po_engine.cu) take the device's SM count, not a literal one."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "pypo_gb300" / "csrc"


def test_no_literal_sm_count():
    code = re.sub(r"//[^\n]*", "", (CSRC / "po_engine.cu").read_text())
    assert not re.findall(r"[^\n]*\b152L?\b[^\n]*", code)

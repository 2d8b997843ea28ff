"""Kernels of a rank round run side by side in the forward graph, and any of them may set a bit of the call's error word
(Ctl::err): every device-side change of it is atomic, or a bit set by another kernel could be lost."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kolmo_gb300", "csrc")


def test_error_word_is_changed_by_atomics_only():
    plain = re.compile(r"(->|\.)err\s*(\|=|&=|\^=|\+=|=(?!=))")
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "fwd*.cu*"))):
        with open(path) as f:
            for no, line in enumerate(f, 1):
                code = line.split("//")[0]
                seen += "err, E_" in code
                assert not plain.search(code), f"{os.path.basename(path)}:{no}: {code.strip()}"
    assert seen > 20  # the sources still name the word so

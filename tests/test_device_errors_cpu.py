"""Kernels on several streams, and many threads of one, report errors in one
word of the device state: every update of it must be an atomic OR, or one
report erases another."""
import os
import re

from conftest import PKG


def test_device_errors_are_or_ed_atomically():
    seen = 0
    csrc = os.path.join(PKG, "csrc")
    for name in sorted(os.listdir(csrc)):
        with open(os.path.join(csrc, name)) as f:
            text = f.read()
        seen += len(re.findall(r"atomicOr\(&a\.ds->err", text))
        plain = re.findall(r"ds->err\s*(?:\|=|=[^=]).*", text)
        assert not plain, (name, plain)
    assert seen >= 8

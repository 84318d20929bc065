"""CPU: the variables and derivative slots that the FP64 constraint kernel prefetches are those
that the generated constraint algebra reads."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sympygr_b200", "csrc")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_prefetched_ranges_are_those_read():
    algebra, kernel = _text("generated/bssn_constraints_algebra.cuh"), _text("constraint_kernels.cuh")
    for table, call in (("kConstraintVars", "u"), ("kConstraintSlots", "d")):
        read = {int(n) for n in re.findall(r"\bin\.%s\((\d+)\)" % call, algebra)}
        ranges = re.search(table + r"\{(\d+), (\d+), (\d+), (\d+)\}", kernel)
        a, b, c, d = (int(n) for n in ranges.groups())
        assert read == set(range(a, b)) | set(range(c, d)), table
        assert "= %s;" % table in kernel

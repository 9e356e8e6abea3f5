"""Which viscosity passes take plain leaves apart, by how many a level has: the
rule of csrc/viscosity_plain.h picks the form that measured faster (or within
the noise of it) for the levels it was measured on."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text('#include "viscosity_plain.h"\nextern "C" {\n'
                   "int restrict_(int nl, int plain) { return uaamg::vplain_restrict(nl, plain); }\n"
                   "int colour(int nl, int plain) { return uaamg::vplain_colour(nl, plain); }\n}\n")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "uaamg_b200", "csrc"), "-o", str(lib),
                    str(src)], check=True)
    return C.CDLL(str(lib))


# leaves, plain leaves, ms of a solve with the lists, without
RESTRICT = [(1107, 245, 6.178, 6.079), (1107, 0, 5.152, 4.984), (1484, 304, 5.317, 5.261), (1484, 0, 5.953, 5.789),
            (1948, 584, 6.466, 6.635), (1948, 440, 6.605, 6.560), (1948, 0, 7.302, 7.161), (2774, 992, 8.771, 8.788),
            (2774, 712, 9.439, 9.435), (2774, 420, 9.821, 9.770), (2774, 0, 10.580, 10.439), (3836, 1172, 11.790, 11.912),
            (3836, 674, 12.485, 12.614), (3836, 480, 13.087, 12.970), (5151, 1976, 14.903, 15.239),
            (5151, 540, 16.663, 16.770), (5151, 216, 19.190, 19.305)]
COLOUR = [(1107, 272, 6.079, 6.097), (1107, 218, 4.738, 4.745), (1107, 120, 4.867, 4.764), (1107, 0, 4.984, 4.804),
          (1484, 334, 5.261, 5.612), (1484, 60, 5.768, 5.826), (1484, 0, 5.789, 5.821), (1948, 192, 6.770, 7.066),
          (1948, 0, 7.161, 7.183), (2774, 1062, 8.788, 9.583), (2774, 210, 10.200, 10.243), (2774, 0, 10.439, 10.332),
          (3836, 272, 13.573, 13.953), (5151, 2084, 15.239, 17.271), (5151, 108, 19.720, 19.777)]


@pytest.mark.parametrize("nl,plain,lists,general", RESTRICT)
def test_restriction(rule, nl, plain, lists, general):
    took, other = (lists, general) if rule.restrict_(nl, plain) else (general, lists)
    assert took <= 1.01 * other


@pytest.mark.parametrize("nl,plain,lists,general", COLOUR)
def test_colour(rule, nl, plain, lists, general):
    took, other = (lists, general) if rule.colour(nl, plain) else (general, lists)
    assert took <= 1.01 * other


def test_no_plain_leaves(rule):
    """What the lists cost where nothing is plain is not paid."""
    for nl in range(1024, 40000, 7):
        assert not rule.restrict_(nl, 0)
        assert nl >= 4096 or not rule.colour(nl, 0)
        assert rule.restrict_(nl, nl) and rule.colour(nl, nl)

"""The rule of the kernels that start under their predecessor: what an earlier kernel of the
chain wrote is not read through the read-only path, which their wait does not order."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "meep_torch_b200", "csrc")
# fields and CPML memory as the kernels name them (descriptors S, split parameters P, adjoint
# buffers B)
CHAIN = r"(?:S\.(?:f_main|f_x|f_y|f|psi)\s*\[|P\.(?:e|eo|h|ho|pi|po|pp|b)\b|B\.(?:g|g_psi|tmp)\s*\[)"


@pytest.mark.parametrize("name", ["yee2d.cu", "yee3d.cu", "adjoint2d.cu", "adjoint3d.cu"])
def test_chain_data_is_not_read_through_the_read_only_path(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    bad = re.findall(r"const float \*\s*__restrict__ \w+ = " + CHAIN + r"[^;]*;", src)
    bad += re.findall(r"(?:__ldg|ldg4v)\(\s*(?:reinterpret_cast<[^>]*>\()?" + CHAIN + r"[^;]*;",
                      src)
    assert not bad, bad

"""CTAs share global memory, so no access to it in the kernels has the scope of one CTA: a load at CTA scope
and another CTA's store are a data race, in which nothing says that a vector is read whole."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "bounce_softbody_gb300", "csrc")


def test_global_memory_is_not_accessed_at_cta_scope():
    found = []
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        found += [(name, m.group(0)) for m in re.finditer(r"\b(?:ld|st|red|atom)\.[\w.:]*\bcta\.global[\w.:]*", text)]
    assert not found

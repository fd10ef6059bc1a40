"""A tree build's first scan writes each node's owner into the buffer of the build before, so it is
bounded by what that buffer holds: the node capacity is raised before the buffers grow, and stays raised
when a growth fails. Read from the source, as provoking it would take a device without free memory."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "galaxy_formation_gb300", "csrc")


def test_the_owners_bound_is_the_size_of_their_buffer():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "gf_tree.cu")).read())
    init = re.search(r"StartScan starts\{(.*?)\};", text, re.S).group(1)
    assert "node_owner.as<int>()" in init
    assert re.search(r"std::min\(size_t\(node_cap\), node_owner\.holds<int>\(\)\)", init)
    # raised only where the buffer has just been grown to it
    grown = text.index("node_owner.get<int>(cap)")
    raised = [m.start() for m in re.finditer(r"starts\.cap = ", text)]
    assert raised and all(grown < at for at in raised)

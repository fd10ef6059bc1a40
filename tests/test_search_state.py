"""The engine's neighbour cache and the visiting order of its search tree hold only after a search that came
through: while one runs (and may throw for lack of memory) neither is marked valid, as the passes that follow
index the particles by them. Read from the source, as provoking it would take a device without free memory."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "galaxy_formation_gb300", "csrc")


def test_cache_and_order_are_invalid_during_a_search():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "gf_hydro.cu")).read())
    start = text.index("if (!have_nb) {")
    search, grow = text.index("knn_exact(", start), text.index("cache.get<int>(", start)
    for name, off, on in (("cache_valid", "cache_valid = false;", "cache_valid = true;"),
                          ("order_ng", "order_ng = -1;", "order_ng = ng;")):
        assert start < text.index(off, start) < min(search, grow), name
        assert text.index(on, start) > search, name
    # the search learns beforehand whether its tree was of this gas set
    assert text.index("same_gas = order_ng == ng", start) < text.index("order_ng = -1;", start)
    call = text[search:text.index(";", search)]
    assert "same_gas" in call and "order_ng" not in call

"""The launch form of a PCG iteration that "auto" takes: by the node count, colour where the incidence does not fit 32 bits."""
from types import SimpleNamespace

import pytest

from difffea_b200.workspace import FUSED_FORM_MAX_NODES, pcg_form_for


@pytest.mark.parametrize("nodes,nen,stride,form", [(4, 4, 32, "fused"), (FUSED_FORM_MAX_NODES - 1, 9, 75_008, "fused"),
                                                   (FUSED_FORM_MAX_NODES, 9, 75_008, "gather"),
                                                   (3_000_000, 3, 6_000_000, "gather"),
                                                   (5 * 10 ** 8, 4, 2 ** 29, "colour"),
                                                   (10, 4, 2 ** 29 - 32, "fused")])
def test_auto_form(nodes, nen, stride, form):
    mesh = SimpleNamespace(n_nodes=nodes, nen=nen, stride=stride, n_el=stride)
    assert pcg_form_for(mesh) == form
    for named in ("colour", "gather", "fused"):
        assert pcg_form_for(mesh, named) == named
    with pytest.raises(ValueError):
        pcg_form_for(mesh, "other")

"""res_calc + bres_calc over corner records with the boundary edges linked in: a second
map from the boundary edges to the nodes (each edge turned round, so its normal too) is
not served by the links of the first."""
import numpy as np
import pytest

from op2b import mesh as M
from op2b.airfoil import Airfoil

pytestmark = pytest.mark.gpu


def _march(op2, turned, **options):
    """One iteration over the mesh's boundary edges, two over `turned` ones (or not)."""
    for k, v in options.items():
        op2.set_option(k, v)
    m = M.channel_bump(61, 37, seed=3)
    app = Airfoil(m)
    app.iterate(1)
    if turned:
        app.pbedge = op2.op_decl_map(app.bedges, app.nodes, 2, np.ascontiguousarray(m.bedge[:, ::-1]),
                                     "pbedge_turned")
        app._build_args()
    app.iterate(2)
    q = app.fetch()["q"]
    op2.op_exit()
    op2.op_init()
    return q


def test_links_of_one_node_map_do_not_serve_another(op2):
    got, plain = _march(op2, True), _march(op2, False)
    want = _march(op2, True, bres_kernel=0)  # every bres_calc a loop of its own
    op2.set_option("bres_kernel", 1)
    assert np.abs(want - plain).max() > 1e-6  # (turning them matters)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()

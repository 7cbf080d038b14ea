"""The plan of the fused step on the CPU: akb_patch_plan_check builds the
patches of a mesh as initFull does and checks every index the kernel will
use."""
import ctypes

import numpy as np
import pytest

import akantu2_b200 as akb
from akantu2_b200 import _capi
from akantu2_b200.mesh import TYPE_IDS


def _check(mesh, max_own, nb_nodes=None):
    L = _capi.lib()
    stats = (ctypes.c_int64 * 4)()
    n = mesh.getNbNodes()
    off = np.array([0, n] if nb_nodes is None else np.concatenate([[0], np.cumsum(nb_nodes)]),
                   dtype=np.int64)
    _capi.check(L.akb_patch_plan_check(TYPE_IDS[mesh.element_type], _capi.ptr(mesh.nodes), n,
                                       _capi.ptr(mesh.connectivity), mesh.getNbElement(),
                                       len(off) - 1, _capi.ptr(off), max_own, stats))
    return list(stats)  # patches, patch elements, largest patch's nodes, and slots


@pytest.mark.parametrize("make", [akb.box_tet4, akb.box_hex8, akb.square_tri6])
@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 5, 6), (19, 3, 8)])
@pytest.mark.parametrize("max_own", [1, 8, 27, 216])
def test_plan_covers_every_node_and_slot(make, cells, max_own):
    cells = cells[:2] if make is akb.square_tri6 else cells
    mesh = make(*cells)
    rng = np.random.default_rng(4)
    for shuffle in (False, True):
        if shuffle:
            new = rng.permutation(mesh.getNbNodes())
            nodes = np.empty_like(mesh.nodes)
            nodes[new] = mesh.nodes
            conn = new[mesh.connectivity][rng.permutation(mesh.getNbElement())]
            mesh = akb.Mesh(mesh.spatial_dimension, nodes, conn.astype(np.int32),
                            mesh.element_type)
        patches, elements, nodes, slots = _check(mesh, max_own)
        assert patches >= mesh.getNbNodes() / max_own and elements >= mesh.getNbElement()
        assert nodes <= mesh.getNbNodes() and slots > 0


def test_plan_keeps_instances_apart_and_isolated_nodes():
    a, b = akb.box_tet4(3), akb.box_tet4(2)
    nodes = np.concatenate([a.nodes, b.nodes, [[5.0, 5.0, 5.0]]])
    conn = np.concatenate([a.connectivity, b.connectivity + a.getNbNodes()])
    mesh = akb.Mesh(3, nodes, conn, "_tetrahedron_4")
    n = [a.getNbNodes(), b.getNbNodes() + 1]
    assert _check(mesh, 27, n)[0] >= 4


def test_regular_grids_are_cut_between_their_planes():
    """a box of 16^3 nodes into patches of 8^3: 8 cubes, each with the 9^3 or
    8^2 x 9 ... elements that touch it"""
    patches, elements, nodes, slots = _check(akb.box_hex8(15), 512)
    assert patches == 8 and elements == 16 ** 3 and nodes == 9 ** 3 and slots == 8 * 512

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


@pytest.mark.parametrize("cells,lengths", [((60, 60, 2), (1, 1, 1)), ((80, 12, 5), (1, 1, 1)),
                                           ((9, 9, 9), (1, 30, 4))])
@pytest.mark.parametrize("max_own", [27, 125, 216])
def test_stretched_cells_are_cut_like_cubic_ones(cells, lengths, max_own):
    """patches hold as many cells along each axis whatever their lengths: the same
    number of patches and of elements evaluated, a twentieth apart"""
    cubic = _check(akb.box_tet4(*cells, lengths=[c / 10 for c in cells]), max_own)
    stretched = _check(akb.box_tet4(*cells, lengths=lengths), max_own)
    for a, b in zip(stretched[:2], cubic[:2]):
        assert abs(a - b) <= b / 20


def test_stretched_instances_of_a_batch():
    """each instance of a batch by its own cells"""
    plate = akb.box_tet4(30, 30, 2)
    cube = akb.box_tet4(7)
    alone = _check(akb.box_tet4(30, 30, 2, lengths=(3.0, 3.0, 0.2)), 125)[1] + _check(cube, 125)[1]
    both = akb.Mesh(3, np.concatenate([plate.nodes, cube.nodes]),
                    np.concatenate([plate.connectivity, cube.connectivity + plate.getNbNodes()]),
                    "_tetrahedron_4")
    got = _check(both, 125, [plate.getNbNodes(), cube.getNbNodes()])[1]
    assert abs(got - alone) <= alone / 20


@pytest.mark.parametrize("n,max_own", [(5, 27), (9, 125), (9, 216)])
def test_plan_of_an_unstructured_mesh(n, max_own):
    """a Delaunay mesh of scattered points: uneven valences, no planes"""
    from scipy.spatial import Delaunay
    points = np.random.default_rng(n).uniform(0, 1, (n ** 3, 3))
    tets = Delaunay(points).simplices
    volume = np.linalg.det(points[tets[:, 1:]] - points[tets[:, :1]])
    tets[volume < 0] = tets[volume < 0][:, [0, 2, 1, 3]]
    mesh = akb.Mesh(3, points, tets.astype(np.int32), "_tetrahedron_4")
    patches, elements, nodes, slots = _check(mesh, max_own)
    assert patches >= n ** 3 / max_own and elements >= len(tets) and slots > 0

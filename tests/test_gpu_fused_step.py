"""The fused step (one launch over patches of nodes) against the two-kernel
step: the same operations in the same order, so the same bits, at the sizes
where its plan can go wrong (one element, one patch, partly filled patches,
meshes whose numbering has no order) and with everything that reaches its
kernel: several materials, an eigen gradient, external forces, blocked dofs,
stopping instances of a batch."""
import numpy as np
import pytest

import akantu2_b200 as akb
from scenarios import (UNIT_ELASTIC, UNIT_NEOHOOKEAN, UNIT_PLASTIC, blocked_face,
                       sinusoidal_velocity)
from test_gpu_parity import gpu_model

pytestmark = pytest.mark.gpu

SVK = dict(UNIT_ELASTIC, finite_deformation=True)
FIELDS = ("getDisplacement", "getVelocity", "getAcceleration", "getInternalForce")


def _shuffled(mesh, seed):
    """the mesh with its nodes and elements renumbered at random"""
    rng = np.random.default_rng(seed)
    new = rng.permutation(mesh.getNbNodes())
    nodes = np.empty_like(mesh.nodes)
    nodes[new] = mesh.nodes
    conn = new[mesh.connectivity][rng.permutation(mesh.getNbElement())]
    return akb.Mesh(mesh.spatial_dimension, nodes, conn.astype(np.int32), mesh.element_type)


def _pair(mesh, mats, precision, mat_of_elem=None, forces=False):
    v0 = sinusoidal_velocity(mesh.nodes, 0.03)
    models = []
    for fused in (True, False):
        m = gpu_model(mesh, mats, mat_of_elem, precision)
        assert m.getFusedStep()
        m.setFusedStep(fused)
        m.setNodal("velocity", v0)
        m.setNodal("blocked_dofs", blocked_face(mesh.nodes))
        if forces:
            m.setNodal("external_force", 1e-3 * np.cos(5 * mesh.nodes) / mesh.getNbNodes())
        m.setTimeStep(0.8 * m.getStableTimeStep())
        models.append(m)
    return models


def _same(models, what=""):
    assert not models[1].getFusedStep()
    for f in FIELDS:
        a, b = (getattr(m, f)() for m in models)
        assert np.isfinite(a).all() and np.array_equal(a, b), (what, f, np.abs(a - b).max())
    assert np.abs(models[0].getInternalForce()).max() > 0


KERNELS = [("_tetrahedron_4", "fp64", UNIT_ELASTIC), ("_tetrahedron_4", "fp64", UNIT_NEOHOOKEAN),
           ("_tetrahedron_4", "fp64", SVK), ("_tetrahedron_4", "mixed", UNIT_ELASTIC),
           ("_tetrahedron_4", "mixed", UNIT_NEOHOOKEAN), ("_tetrahedron_4", "mixed", SVK),
           ("_hexahedron_8", "mixed", UNIT_ELASTIC), ("_hexahedron_8", "mixed", UNIT_NEOHOOKEAN),
           ("_hexahedron_8", "mixed", SVK)]


def _box(etype, *cells):
    return (akb.box_tet4 if etype == "_tetrahedron_4" else akb.box_hex8)(*cells)


@pytest.mark.parametrize("etype,precision,mat", KERNELS)
@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 6, 5), (23, 9, 17)])
def test_fused_step_is_bit_identical(etype, precision, mat, cells):
    models = _pair(_box(etype, *cells), [mat], precision, forces=cells[0] == 7)
    for steps in (1, 130, 2):  # eager, a graph with a tail, eager again
        for m in models:
            m.solveStep(steps)
        _same(models, steps)
    assert all(m.getStatus() == 0 for m in models)


@pytest.mark.parametrize("etype,precision,mat", KERNELS)
def test_fused_step_of_a_shuffled_mesh_with_two_materials(etype, precision, mat):
    mesh = _shuffled(_box(etype, 9, 8, 7), 3)
    soft = dict(mat, name="soft", E=0.5, nu=0.2, eigen_grad_u=[[1e-3, 0, 0], [0, 2e-3, 0],
                                                               [5e-4, 0, 0]])
    which = (np.arange(mesh.getNbElement()) % 3 == 0).astype(np.int32)
    models = _pair(mesh, [mat, soft], precision, mat_of_elem=which)
    for m in models:
        m.solveStep(120)
    _same(models)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fused_step_of_a_distorted_tetrahedral_mesh(precision):
    mesh = akb.box_tet4(11, 5, 8)
    x = mesh.nodes
    inner = np.all((x > 1e-9) & (x < 1 - 1e-9), axis=1)
    x[inner] += np.random.default_rng(1).uniform(-0.02, 0.02, (inner.sum(), 3))
    models = _pair(_shuffled(mesh, 8), [UNIT_NEOHOOKEAN], precision)
    for m in models:
        m.solveStep(110)
    _same(models)


@pytest.mark.parametrize("etype,precision,mat", KERNELS[::2])
def test_fused_batch_with_stopping_instances(etype, precision, mat):
    runs = []
    for fused in (True, False):
        b = akb.BatchModel([_box(etype, n) for n in (2, 7, 4)])
        for k in range(3):
            b.addMaterial(mat["type"], **{**{k_: v for k_, v in mat.items() if k_ != "type"},
                                          "name": f"m{k}", "E": 1.0 + 0.3 * k})
        b.setInstanceMaterials(np.arange(3))
        b.initFull(precision=precision)
        assert b.getFusedStep()
        b.setFusedStep(fused)
        b.setTimeSteps(0.8 * b.getStableTimeSteps())
        b.setNodal("velocity", sinusoidal_velocity(b.mesh.nodes, 0.03))
        b.setNodal("blocked_dofs", blocked_face(b.mesh.nodes))
        b.setInstanceSteps([30, 150, 77])
        b.solveStep(160)
        runs.append([getattr(b, f)() for f in FIELDS[:3]])
    for f, x, y in zip(FIELDS, *runs):
        assert np.isfinite(x).all() and np.abs(x).max() > 0 and np.array_equal(x, y), f


def test_fused_step_rules():
    """which models have it, and which settings leave it"""
    m = gpu_model(akb.box_tet4(3), [UNIT_ELASTIC], precision="mixed")
    assert m.getFusedStep()
    m.setNodeShape(256, 0)
    assert not m.getFusedStep()
    m.setFusedStep(True)
    m.setLaunchShape("elastic", 64, 8, 128)
    assert not m.getFusedStep()
    two = gpu_model(akb.box_tet4(3), [UNIT_ELASTIC, dict(UNIT_PLASTIC)],
                    (np.arange(162) % 2).astype(np.int32), "mixed")
    assert not two.getFusedStep()
    with pytest.raises(akb.AkbError) as e:
        two.setFusedStep(True)
    assert e.value.name == "AKB_EUNSUPPORTED"


def test_internal_force_across_a_change_of_step_form():
    """the internal force of the last step is there whichever form made it"""
    mesh = akb.box_tet4(5)
    models = _pair(mesh, [UNIT_NEOHOOKEAN], "mixed")
    for m in models:
        m.solveStep(3)
    models[1].setFusedStep(True)
    models[0].setFusedStep(False)
    a, b = (m.getInternalForce() for m in models)
    assert np.abs(a).max() > 0 and np.array_equal(a, b)
    for m in models:
        m.solveStep(101)
    _same(models[::-1])


def _plastic_pair(nx, ny, precision, rule, shuffle=None, mats=(UNIT_PLASTIC,), which=None):
    mesh = akb.square_tri6(nx, ny)
    if shuffle is not None:
        mesh = _shuffled(mesh, shuffle)
    x = mesh.nodes
    v0 = 0.02 * np.stack([np.sin(3 * x[:, 0]), np.cos(2 * x[:, 1])], axis=1) * x[:, :1]
    models = []
    for fused in (True, False):
        m = gpu_model(mesh, list(mats), which, precision, rule)
        assert m.getFusedStep()
        m.setFusedStep(fused)
        m.setNodal("velocity", v0)
        m.setNodal("blocked_dofs", blocked_face(x, axis=0))
        m.setTimeStep(0.8 * m.getStableTimeStep())
        m.setPrescribedVelocityRamp(np.isclose(x[:, 0], 1.0), 0, 5e-3, 50)
        models.append(m)
    return models


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("cells,shuffle", [((1, 1), None), ((9, 7), None), ((31, 18), 5)])
def test_fused_plastic_triangles_are_bit_identical(precision, rule, cells, shuffle):
    soft = dict(UNIT_PLASTIC, name="soft", E=0.6, sigma_y=5e-4, h=0.2)
    which = (np.arange(2 * cells[0] * cells[1]) % 3 == 0).astype(np.int32)
    models = _plastic_pair(*cells, precision, rule, shuffle, (UNIT_PLASTIC, soft), which)
    for steps in (1, 130, 2):
        for m in models:
            m.solveStep(steps)
        _same(models, steps)
        for k in range(2):
            for f in ("stress", "grad_u", "inelastic_strain", "iso_hardening", "plastic_energy"):
                a, b = (m.getMaterial(k).getInternal(f)() for m in models)
                assert np.array_equal(a, b), (k, f)
    assert models[0].getMaterial(0).getInternal("iso_hardening")().max() > 0, "must yield"


def test_fused_heated_plastic_triangles():
    """the thermal term of the first step reaches the fused kernel"""
    models = _plastic_pair(6, 5, "mixed", 0, mats=(dict(UNIT_PLASTIC, alpha=1e-4, delta_T=5.0),))
    for m in models:
        m.solveStep(105)
    _same(models)


@pytest.mark.parametrize("precision,cells", [("fp64", (57, 59, 58)), ("mixed", (67, 69, 68))])
def test_fused_step_whose_tables_are_larger_than_l2(precision, cells):
    """patches that prefetch the next wave's tables, up to the last one"""
    models = _pair(_box("_tetrahedron_4", *cells), [UNIT_ELASTIC], precision)
    for m in models:
        m.solveStep(5)
    _same(models)


@pytest.mark.parametrize("n", [36, 38, 43])
def test_dependent_launches_around_one_wave(n):
    """two-kernel steps whose kernels are resident together, not quite, and of
    more than one wave: with and without dependent launches the same bits, with a
    setting changed between two sequences"""
    mesh = akb.box_hex8(n)
    models = []
    for dependent in (True, False):
        m = gpu_model(mesh, [UNIT_NEOHOOKEAN], precision="mixed")
        assert not m.getFusedStep()
        m.setDependentLaunch(dependent)
        m.setNodal("velocity", sinusoidal_velocity(mesh.nodes, 0.03))
        m.setTimeStep(0.8 * m.getStableTimeStep())
        m.solveStep(103)
        m.setNodeShape(64, 0)
        m.solveStep(2)
        models.append(m)
    _same(models)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_internal_force_of_stopped_instances(precision, fused):
    """an instance that stops at once, in the middle of a sequence or with its
    last step has the internal force of its own last step, in both forms of the
    step: that of the same mesh run alone"""
    meshes = [akb.box_tet4(n) for n in (3, 6, 4)]
    b = akb.BatchModel(meshes)
    mat = {k: v for k, v in UNIT_ELASTIC.items() if k != "type"}
    b.addMaterial("elastic", **mat)
    b.initFull(precision=precision)
    b.setFusedStep(fused)
    dt = 0.8 * b.getStableTimeSteps()
    b.setTimeSteps(dt)
    b.setNodal("velocity", sinusoidal_velocity(b.mesh.nodes, 0.03))
    b.solveStep(20)
    b.setInstanceSteps([0, 30, 7])
    b.solveStep(30)
    b.solveStep(5)
    for k, steps in enumerate((20, 50, 27)):
        alone = gpu_model(meshes[k], [UNIT_ELASTIC], precision=precision)
        alone.setNodal("velocity", sinusoidal_velocity(meshes[k].nodes, 0.03))
        alone.setTimeStep(float(dt[k]))
        alone.solveStep(steps)
        for f in FIELDS:
            a, c = getattr(b, f)()[b.instance_nodes(k)], getattr(alone, f)()
            assert np.abs(c).max() > 0 and np.array_equal(a, c), (k, f)


@pytest.fixture
def device_limit():
    """limits the device bytes of this thread's models, as a smaller device"""
    from akantu2_b200 import _capi

    def limit(nbytes):
        _capi.check(_capi.lib().akb_debug_limit_device_bytes(int(nbytes)))

    yield limit
    limit(0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_without_memory_for_the_plan_the_two_kernels_step(device_limit, precision):
    """a device with room for the model but not for the fused step's plan"""
    mesh = akb.box_tet4(6)
    full = gpu_model(mesh, [UNIT_ELASTIC], precision=precision)
    assert full.getFusedStep()
    device_limit(1)
    with pytest.raises(akb.AkbError) as e:
        gpu_model(mesh, [UNIT_ELASTIC], precision=precision)
    assert e.value.name == "AKB_ENOMEM"
    device_limit(full.getDeviceBytes() - 1)
    m = gpu_model(mesh, [UNIT_ELASTIC], precision=precision)
    assert not m.getFusedStep() and m.getDeviceBytes() < full.getDeviceBytes()
    device_limit(0)
    dt = 0.8 * full.getStableTimeStep()
    for x in (full, m):
        x.setNodal("velocity", sinusoidal_velocity(mesh.nodes, 0.03))
        x.setTimeStep(dt)
        x.solveStep(130)
    _same([full, m])


def test_the_plan_gives_its_memory_back(device_limit):
    """what a model asks for later comes before its plan: the same steps go on
    as two kernels"""
    mesh = akb.box_tet4(6)
    models = _pair(mesh, [UNIT_ELASTIC], "fp64")
    for m in models:
        m.solveStep(130)
    device_limit(models[0].getDeviceBytes())
    models[0].setIncrementTracking(True)
    device_limit(0)
    assert not models[0].getFusedStep()
    models[1].setIncrementTracking(True)
    for m in models:
        m.solveStep(130)
    _same(models)
    a, b = (m.getPreviousDisplacement() for m in models)
    assert np.array_equal(a, b)


def test_a_ramp_that_cannot_be_set_leaves_the_model_as_it_was(device_limit):
    """without memory for its buffers the call fails; the steps that follow are
    those of the model without it, or with the ramp it had"""
    mesh = akb.box_tet4(6)
    top = np.isclose(mesh.nodes[:, 2], 1.0)
    for earlier in (False, True):
        models = []
        for failing in (True, False):
            m = gpu_model(mesh, [UNIT_ELASTIC], precision="fp64")
            m.setNodal("velocity", sinusoidal_velocity(mesh.nodes, 0.03))
            m.setNodal("blocked_dofs", blocked_face(mesh.nodes))
            m.setTimeStep(0.8 * m.getStableTimeStep())
            if earlier:
                m.setPrescribedVelocityRamp(top, 1, 1e-2, 10)
            m.solveStep(5)
            if failing:
                device_limit(1)
                with pytest.raises(akb.AkbError):
                    m.setPrescribedVelocityRamp(top, 0, 5e-2, 20)
                device_limit(0)
            m.solveStep(130)
            models.append(m)
        for f in FIELDS + ("getBlockedDOFs",):
            a, b = (getattr(m, f)() for m in models)
            assert np.array_equal(a, b), (earlier, f)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cells,count,fused", [(1, 100, True), (1, 2000, False), (2, 2000, False),
                                               (4, 300, True)])
def test_batches_of_tiny_instances_step_as_two_kernels(precision, cells, count, fused):
    """an instance is a patch at least: many of a few elements are rounds of
    nearly empty blocks"""
    b = akb.BatchModel([akb.box_tet4(cells)] * count)
    b.addMaterial("elastic", rho=1.0, E=1.0, nu=0.3)
    b.initFull(precision=precision)
    assert b.getFusedStep() == fused


@pytest.mark.parametrize("cells,fused", [((100, 100), True), ((400, 20), False)])
def test_triangles_whose_patches_are_not_resident_step_as_two_kernels(cells, fused):
    m = gpu_model(akb.square_tri6(*cells), [UNIT_PLASTIC], precision="mixed")
    assert m.getFusedStep() == fused


@pytest.mark.parametrize("mat,n,dependent", [(UNIT_ELASTIC, 9, True), (UNIT_PLASTIC, 9, True),
                                             (UNIT_PLASTIC, 20, True), (UNIT_NEOHOOKEAN, 9, True),
                                             (UNIT_NEOHOOKEAN, 20, False),
                                             (UNIT_NEOHOOKEAN, 28, True),
                                             (UNIT_NEOHOOKEAN, 35, False)])
def test_dependent_launches_of_fp64_hexahedra(mat, n, dependent):
    """on but for the neohookean law at one to four and eight to twelve blocks per
    SM; the setting changes no result"""
    mesh = akb.box_hex8(n)
    runs = []
    for other in (False, True):
        m = gpu_model(mesh, [mat])
        assert m.getDependentLaunch() == dependent
        m.setDependentLaunch(dependent != other)
        m.setNodal("velocity", sinusoidal_velocity(mesh.nodes, 0.03))
        m.setTimeStep(0.8 * m.getStableTimeStep())
        m.solveStep(103)
        runs.append(m.getDisplacement())
    assert np.abs(runs[0]).max() > 0 and np.array_equal(*runs)


@pytest.mark.parametrize("cells", [(36, 32, 21), (44, 36, 22)])
def test_timing_the_forms_leaves_the_model_at_rest(cells):
    """sizes at which initFull times both forms of the step: the model is at
    rest afterwards, forces of an eigen gradient included, and steps as one that
    was told to use two kernels"""
    mesh = akb.box_tet4(*cells, lengths=[c / 40 for c in cells])
    mat = dict(UNIT_ELASTIC, eigen_grad_u=[[1e-3, 0, 0], [0, 2e-3, 0], [5e-4, 0, 0]])
    models = []
    for two in (False, True):
        m = gpu_model(mesh, [mat], precision="mixed")
        for f in FIELDS:
            x = getattr(m, f)()
            assert not x.any() and not np.signbit(x).any(), f
        assert m.getStatus() == 0
        if two:
            m.setNodeShape(*m.getNodeShape())  # leaves the fused step
        m.setTimeStep(0.8 * m.getStableTimeStep())
        m.solveStep(3)
        models.append(m)
    _same(models)

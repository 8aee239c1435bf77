"""The two-pass step kernels and the reverse step's two passes against the NumPy oracle: every way they are launched (launches
per pass, one cluster, one cooperative launch), at row lengths around the 16-byte groups, and with more than two CPML slabs on an axis (the
row-table path). Bars: fields, CPML memories and traces bitwise, like the other step kernels (same operations, same
order, no contraction); gradients within the relative L2 of tests/test_gpu_adjoint.py."""
from dataclasses import replace

import numpy as np
import pytest

from oracle.adjoint_oracle import AdjointOracle
from oracle.yee_oracle import YeeOracle
from torchfdtd_b200 import Project, Region
from torchfdtd_b200.models import BoundaryFace, Monitor, Source
from torchfdtd_b200.plan import plan_grid

pytestmark = pytest.mark.gpu


def scene(shape, precision, faces=None, component='Ey', steps=12):
    two_d = shape[2] == 1
    region = Region(dimension='2d' if two_d else '3d', size=tuple(n * .05 for n in shape[:2]) + (1 if two_d else shape[2] * .05,),
                    mesh=.05, pml_cells=4, steps=steps, precision=precision, backend='cuda')
    for name, face in (faces or {}).items():
        setattr(region.boundaries, name, face)
    return Project(region=region, sources=[Source(center=(.1, 0, 0), component=component, pulse_cycles=1, wavelength=.6)],
                   monitors=[Monitor(center=(-.1, .05, 0), component=component)])


def assert_matches_oracle(plan, seed, kernel='gather', launches=None):
    from torchfdtd_b200.native import NativeGrid
    rng = np.random.default_rng(seed)
    oracle = YeeOracle(plan)
    advanced = plan.active_components()
    for family, field in (('E', oracle.E), ('H', oracle.H)):
        for c in range(3):
            if family + 'xyz'[c] in advanced:
                field[..., c] = rng.normal(size=plan.shape).astype(plan.dtype)
    grid = NativeGrid(plan, kernel=kernel)
    assert launches is None or grid.step_launches(5) == launches
    grid.set_fields(oracle.E, oracle.H)
    grid.step(5)
    grid.step(plan.steps - 5)
    oracle.run()
    E, H = grid.get_fields()
    np.testing.assert_array_equal(E, oracle.E)
    np.testing.assert_array_equal(H, oracle.H)
    np.testing.assert_array_equal(grid.get_traces(), oracle.traces)
    for got, want in zip(grid.get_psi(), oracle.memory_states):
        np.testing.assert_array_equal(got, want)
    assert grid.counter() == plan.steps and grid.device_status() == 0
    grid.close()


PERIODIC_Y = {'y_min': BoundaryFace(kind='periodic'), 'y_max': BoundaryFace(kind='periodic')}


@pytest.mark.parametrize('mode', ['0', '1', '2'])
@pytest.mark.parametrize('shape,precision,faces,component', [
    ((13, 14, 15), 'float32', None, 'Ey'), ((14, 13, 16), 'float64', {'z_max': BoundaryFace(kind='pec')}, 'Hz'),
    ((32, 13, 14), 'float32', PERIODIC_Y, 'Ez'), ((65, 33, 1), 'float32', PERIODIC_Y, 'Hz'), ((67, 40, 1), 'float64', None, 'Ex')])
def test_every_launch_form_matches_the_oracle(monkeypatch, mode, shape, precision, faces, component):
    monkeypatch.setenv('TFD_PASS_STEPS', mode)
    assert_matches_oracle(plan_grid(scene(shape, precision, faces, component)), 3, launches=10 if mode == '0' else 1)


@pytest.mark.parametrize('precision', ['float32', 'float64'])
def test_more_than_two_slabs_on_an_axis(precision):
    plan = plan_grid(scene((21, 18, 16), precision))
    segments = []                                       # x slabs in two parts each; no z slabs (12 segments at most)
    for s in plan.segments:
        cut = (s.lo + s.hi) // 2 if s.axis == 0 else s.hi
        for lo, hi in ((s.lo, cut), (cut, s.hi)):
            if lo < hi and s.axis < 2:
                part = slice(lo - s.lo, hi - s.lo)
                segments.append(replace(s, lo=lo, hi=hi, b=s.b[part], c=s.c[part], inv_kappa=s.inv_kappa[part]))
    assert len(segments) == 12
    assert_matches_oracle(replace(plan, segments=segments), 4)


@pytest.mark.parametrize('shape,steps', [((40, 30, 20), 3), ((24, 22, 260), 2)])
def test_default_3d_step_equals_the_marching_kernel(shape, steps):
    from torchfdtd_b200.native import NativeGrid
    plan = plan_grid(scene(shape, 'float32', steps=10))
    rng = np.random.default_rng(1)
    start = [rng.normal(size=(*plan.shape, 3)).astype(np.float32) for _ in range(2)]
    out = []
    for variant in (0, 14):
        grid = NativeGrid(plan, variant=variant)
        assert grid.kernel == ('march' if variant else 'gather')
        grid.set_fields(*start)
        grid.step(steps)
        out.append((*grid.get_fields(), *grid.get_psi()))
        grid.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize('shape,precision,faces,component', [
    ((13, 14, 15), 'float32', None, 'Ey'), ((14, 13, 16), 'float64', {'z_max': BoundaryFace(kind='pec')}, 'Hz'),
    ((17, 15, 13), 'float64', {**PERIODIC_Y, 'x_max': BoundaryFace(kind='pec')}, 'Ez'),
    ((15, 16, 13), 'float64', {'x_min': BoundaryFace(kind='periodic'), 'x_max': BoundaryFace(kind='periodic')}, 'Ez'),
    ((65, 33, 1), 'float32', PERIODIC_Y, 'Hz'), ((34, 40, 1), 'float64', None, 'Ez')])
def test_reverse_step_matches_the_oracle(shape, precision, faces, component):
    import torch
    from torchfdtd_b200.adjoint import DifferentiableSimulation
    project = scene(shape, precision, faces, component, steps=24)
    plan = plan_grid(project)
    rng = np.random.default_rng(8)
    eps = rng.uniform(1, 3, size=plan.shape)
    w = rng.normal(size=(plan.steps, 1))
    dtype = torch.float32 if precision == 'float32' else torch.float64
    model = DifferentiableSimulation(project)
    epsilon = torch.tensor(eps, dtype=dtype, device='cuda', requires_grad=True)
    result = model(epsilon)
    (result.signals * torch.tensor(w, dtype=dtype, device='cuda')).sum().backward()
    oracle = AdjointOracle(plan, eps.astype(plan.dtype))
    np.testing.assert_array_equal(result.signals.detach().cpu().numpy(), oracle.forward())
    want = oracle.backward(w.astype(plan.dtype))
    got = epsilon.grad.cpu().numpy()
    assert np.linalg.norm(got - want) <= (1e-5 if precision == 'float32' else 1e-11) * np.linalg.norm(want) and np.linalg.norm(want) > 0
    model.close()


@pytest.mark.parametrize('mode', ['1', '2'])
def test_a_launch_runs_at_most_2_20_steps(monkeypatch, mode):
    """The cooperative form's barrier counts every arrival of a launch in 32 bits: 2^31 - 1 steps in one launch on 148 CTAs would
    pass 2^32 arrivals. Counted, not run."""
    from torchfdtd_b200.native import NativeGrid
    monkeypatch.setenv('TFD_PASS_STEPS', mode)
    grid = NativeGrid(plan_grid(scene((13, 14, 15), 'float32')), kernel='gather')
    assert [grid.step_launches(n) for n in (0, 1, 1 << 20, (1 << 20) + 1, 2**31 - 1)] == [0, 1, 1, 2, 2048]
    grid.close()


def dispersive(project):
    """A Drude rod through the middle of the grid."""
    from torchfdtd_b200 import Material, Structure
    extra = dict(materials=[Material(name='metal', model='drude', epsilon_inf=1.5, plasma_rad_s=9e15, collision_rad_s=1e14)],
                 structures=[Structure(size=(.2, .2, project.region.size[2]), center=(.1, 0, 0), material='metal')])
    return Project(region=project.region, sources=project.sources, monitors=project.monitors, **extra)


@pytest.mark.parametrize('mode', ['0', '1', '2'])
@pytest.mark.parametrize('name,precision', [('plain', 'float32'), ('tmz', 'float64'), ('dispersive', 'float64'), ('tfsf', 'float32'), ('tfsf', 'float64')])
def test_adjoint_segment_equals_its_steps_one_by_one(monkeypatch, name, precision, mode):
    """tfd_adjoint_segment against save, step and tfd_adjoint_step, bitwise. Both start from a reset plan: a restart state holds
    neither a TFSF box's incident line nor pole states."""
    import torch
    from torchfdtd_b200.native import NativeAdjoint, NativeGrid
    monkeypatch.setenv('TFD_PASS_STEPS', mode)
    project = scene((21, 22, 1) if name == 'tmz' else (21, 22, 23), precision, component='Ez' if name == 'tmz' else 'Ey', steps=14)
    if name == 'dispersive':
        project = dispersive(project)
    if name == 'tfsf':
        box = Source(kind='tfsf', normal='x', direction='+', size=(.4, .4, .4), component='Ey', pulse_cycles=1, wavelength=.6)
        project = Project(region=project.region, sources=[box], monitors=project.monitors)
    plan = plan_grid(project)
    assert bool(plan.tfsf) == (name == 'tfsf')
    grid = NativeGrid(plan, kernel='gather')
    adjoint = NativeAdjoint(grid)
    count = 12
    seeds = torch.tensor(np.random.default_rng(5).normal(size=(count, 1)), dtype=grid.torch_dtype, device='cuda')
    slots = torch.zeros((count, grid.state_bytes()), dtype=torch.uint8, device='cuda')
    replay, checkpoint = torch.zeros_like(slots), torch.zeros_like(slots[0])
    grid.reset()
    grid.save_state(checkpoint)
    for j in range(count):
        grid.save_state(slots[j])
        grid.step(1)
    for j in range(count - 1, -1, -1):
        adjoint.step(slots[j], seeds[j].contiguous())
    want = adjoint.sensitivity().clone()
    grid.reset()
    adjoint.reset()
    adjoint.segment(checkpoint, count, replay, seeds)
    got = adjoint.sensitivity()
    assert want.abs().max() > 0
    np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())
    adjoint.close()
    grid.close()


def test_kernel_name_is_the_kernel_that_steps(monkeypatch):
    """NativeGrid.kernel and the launches of a step: a kernel asked for by name runs, 'auto' names its choice ('tile2d': any of
    the 2D TMz forms)."""
    from torchfdtd_b200.native import NativeGrid
    flat = scene((48, 44, 1), 'float32', component='Ez')
    monkeypatch.setenv('TFD_PASS_STEPS', '0')
    got = []
    for project, kernel, env in ((scene((21, 18, 16), 'float32'), 'auto', {}), (scene((21, 18, 16), 'float32'), 'march', {}),
                                 (scene((21, 18, 16), 'float64'), 'march', {}), (flat, 'auto', {}),
                                 (flat, 'tile2d', {'TFD_CLUSTER2D': '0'}), (flat, 'tile2d', {'TFD_CLUSTER2D': '0', 'TFD_PERSIST2D': '0'})):
        for k in ('TFD_CLUSTER2D', 'TFD_PERSIST2D'):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        grid = NativeGrid(plan_grid(project), kernel=kernel)
        got.append((grid.kernel, grid.step_launches(4)))
        grid.close()
    assert [k for k, _ in got] == ['gather', 'march', 'march', 'tile2d', 'tile2d', 'tile2d']
    assert got[0][1] == 8 and got[3][1] == 1 and got[4][1] == 8 and all(n <= 12 for _, n in got)


@pytest.mark.parametrize('mode', ['0', '1', '2'])
@pytest.mark.parametrize('shape,precision,frequencies', [((21, 18, 16), 'float32', 1), ((21, 18, 16), 'float64', 7), ((40, 36, 1), 'float32', 257)])
def test_plane_accumulators_of_any_frequency_count(monkeypatch, shape, precision, frequencies, mode):
    """DFT planes of the one-launch forms and of a launch per step, below, at and past the chunks of frequencies that one
    pass over the accumulators takes; the double-precision sums of the CPU oracle to 1e-12."""
    from oracle.cpu import CpuOracle
    from torchfdtd_b200 import FieldMonitor, SpectrumSettings
    from torchfdtd_b200.native import NativeGrid
    monkeypatch.setenv('TFD_PASS_STEPS', mode)
    project = scene(shape, precision, component='Hz' if shape[2] == 1 else 'Ey', steps=13)
    spectrum = SpectrumSettings(sampling='frequency', frequency_points=frequencies, apodization='none')
    plane = FieldMonitor(normal='x', center=(.1, 0, 0), size=(0, .3, 1 if shape[2] == 1 else .2), dft_precision='float64', spectrum=spectrum)
    plan = plan_grid(Project(region=project.region, sources=project.sources, monitors=[plane]))
    want = CpuOracle(plan).run_with_planes(dft_float64=True)
    grid = NativeGrid(plan, kernel='gather')
    grid.step(6)
    grid.step(7)
    got = grid.get_plane(0)
    assert got.shape[0] == frequencies and np.abs(got).max() > 0
    assert np.linalg.norm(got - want[0]) <= 1e-12 * np.linalg.norm(want[0])
    grid.close()


@pytest.mark.parametrize('shape,precision,plane', [
    ((21, 18, 16), 'float32', False), ((21, 18, 16), 'float64', True), ((42, 37, 30), 'float32', False), ((42, 37, 30), 'float32', True),
    ((70, 66, 72), 'float32', True), ((90, 100, 103), 'float64', False), ((103, 90, 1), 'float32', True), ((103, 90, 1), 'float64', True)])
def test_calls_of_any_length_match_the_oracle(shape, precision, plane):
    """The default launch form of short and long calls on one plan: one cluster, one cooperative launch of one, two (moved on
    from sweep to sweep) and more than six sweeps, strips in one launch, launches per pass."""
    from oracle.cpu import CpuOracle
    from torchfdtd_b200 import FieldMonitor, SpectrumSettings
    from torchfdtd_b200.native import NativeGrid
    two_d = shape[2] == 1
    project = scene(shape, precision, component='Ez' if two_d else 'Ey', steps=14)
    if plane:
        spectrum = SpectrumSettings(sampling='frequency', frequency_points=3, apodization='none')
        monitor = FieldMonitor(normal='y', center=(0, .1, 0), size=(.4, 0, 1 if two_d else .2), dft_precision='float64', spectrum=spectrum)
        project = Project(region=project.region, sources=project.sources, monitors=[*project.monitors, monitor])
    plan = plan_grid(project)
    oracle = CpuOracle(plan)
    grid = NativeGrid(plan)
    want = oracle.run_with_planes(dft_float64=True)
    for count in (1, 4, 2, 3, 20):
        grid.step(count)
    E, H = grid.get_fields()
    np.testing.assert_array_equal(E, oracle.E)
    np.testing.assert_array_equal(H, oracle.H)
    np.testing.assert_array_equal(grid.get_traces(), oracle.traces)
    for got, expected in zip(grid.get_psi(), oracle.memory_states):
        np.testing.assert_array_equal(got, expected)
    for k, value in enumerate(want):
        assert np.linalg.norm(grid.get_plane(k) - value) <= 1e-12 * np.linalg.norm(value) and np.linalg.norm(value) > 0
    assert grid.counter() == plan.steps and grid.device_status() == 0
    grid.close()


def test_pole_states_do_not_depend_on_the_order_of_the_samples():
    """The library numbers a state's samples in memory order: any order of the caller's gives the same run, a sample listed
    twice or by two states is refused."""
    from torchfdtd_b200.native import NativeGrid
    plan = plan_grid(dispersive(scene((21, 22, 23), 'float32')))
    state = plan.ade[0]
    assert len(plan.ade) == 1 and state.samples > 100
    order = np.random.default_rng(2).permutation(state.samples)
    half = state.samples // 2
    out = []
    halves = [replace(state, target=state.target[half:]), replace(state, target=state.target[:half])]
    for ade in ([state], [replace(state, target=state.target[order])], halves):
        grid = NativeGrid(replace(plan, ade=ade))
        grid.step(plan.steps)
        out.append((*grid.get_fields(), np.array(grid.diagnose())))
        grid.close()
    for other in out[1:]:
        for a, b in zip(out[0][:2], other[:2]):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_allclose(other[2], out[0][2], rtol=1e-12)
    for ade in ([replace(state, target=np.append(state.target[:-1], state.target[0]))], [state, replace(state, target=state.target[5:6])]):
        with pytest.raises(ValueError, match='overlap'):
            NativeGrid(replace(plan, ade=ade))


@pytest.mark.parametrize('mode,launches', [('0', 15), ('2', 1)])
@pytest.mark.parametrize('precision', ['float32', 'float64'])
def test_dispersive_sweep_matches_the_oracle(monkeypatch, precision, mode, launches):
    """The sweep over the dispersive samples as a launch of its own (the form of every large plan) and inside the one launch; the
    source drives some of the samples."""
    monkeypatch.setenv('TFD_PASS_STEPS', mode)
    assert_matches_oracle(plan_grid(dispersive(scene((21, 22, 23), precision))), 6, launches=launches)


@pytest.mark.parametrize('shape,precision,component,metal', [
    ((13, 14, 15), 'float32', 'Ey', False), ((14, 13, 16), 'float64', 'Hz', False), ((65, 33, 1), 'float32', 'Hz', False),
    ((21, 22, 23), 'float32', 'Ey', True)])
def test_64_bit_index_variant_matches_the_oracle(monkeypatch, shape, precision, component, metal):
    """The kernels of arrays of 2^31 elements and more, at a size that a test can hold."""
    monkeypatch.setenv('TFD_PASS_WIDE', '1')
    project = scene(shape, precision, component=component)
    assert_matches_oracle(plan_grid(dispersive(project) if metal else project), 7, launches=15 if metal else 10)


def test_planes_past_65535_match_the_oracle(monkeypatch):
    """A pass walks the planes that its launch grid cannot number."""
    from oracle.cpu import CpuOracle
    from torchfdtd_b200.native import NativeGrid
    monkeypatch.setenv('TFD_PASS_STEPS', '0')
    project = scene((13, 13, 65700), 'float32', steps=10)
    project.sources[0].center = (.1, 0, 1635.0)
    plan = plan_grid(project)
    assert plan.shape == (13, 13, 65700)
    grid = NativeGrid(plan, kernel='gather')
    rng = np.random.default_rng(4)
    oracle = CpuOracle(plan)
    oracle.E[:] = rng.normal(size=oracle.E.shape).astype(np.float32)
    grid.set_fields(oracle.E, oracle.H)
    grid.step(4)
    oracle.run(4)
    E, H = grid.get_fields()
    np.testing.assert_array_equal(E, oracle.E)
    np.testing.assert_array_equal(H, oracle.H)
    grid.close()


@pytest.mark.parametrize('wide', [False, True])
@pytest.mark.parametrize('precision', ['float32', 'float64'])
def test_reverse_step_variants_match_the_oracle(monkeypatch, precision, wide):
    """A grid with plain rows, rows near a face or slab and groups near an x slab: each variant of the reverse step's passes."""
    import torch
    from torchfdtd_b200.adjoint import DifferentiableSimulation
    if wide:
        monkeypatch.setenv('TFD_PASS_WIDE', '1')
    project = scene((40, 24, 22), precision, steps=20)
    plan = plan_grid(project)
    rng = np.random.default_rng(12)
    eps, w = rng.uniform(1, 3, size=plan.shape), rng.normal(size=(plan.steps, 1))
    dtype = torch.float32 if precision == 'float32' else torch.float64
    model = DifferentiableSimulation(project)
    epsilon = torch.tensor(eps, dtype=dtype, device='cuda', requires_grad=True)
    (model(epsilon).signals * torch.tensor(w, dtype=dtype, device='cuda')).sum().backward()
    oracle = AdjointOracle(plan, eps.astype(plan.dtype))
    oracle.forward()
    want = oracle.backward(w.astype(plan.dtype))
    assert np.linalg.norm(epsilon.grad.cpu().numpy() - want) <= (1e-5 if precision == 'float32' else 1e-11) * np.linalg.norm(want)
    assert np.linalg.norm(want) > 0
    model.close()


@pytest.mark.parametrize('shape,sampling,kernel', [((512, 512, 128), 'cell', 'march'), ((256, 256, 512), 'cell', 'gather'),
                                                   ((512, 512, 126), 'cell', 'gather'), ((512, 512, 128), 'yee', 'gather')])
def test_default_kernel_of_large_uniform_grids(shape, sampling, kernel):
    """The marching kernel from 2^25 cells on where the grid fills its tiles; the bitwise equality of both at such a size is
    tests/test_gpu_configs.py's."""
    import torch
    from torchfdtd_b200.native import NativeGrid
    project = scene(shape, 'float32')
    project.region.material_sampling = sampling
    plan = plan_grid(project, material=False)
    plan.epsilon, plan.inv_eps = torch.ones(plan.shape if sampling == 'cell' else (*plan.shape, 3), device='cuda'), None
    grid = NativeGrid(plan, material=plan.epsilon)
    assert grid.kernel == kernel
    grid.close()

"""What the engine is asked to do, as timed cases: resident plans stepped over their range of sizes, boundaries,
precisions and materials, an uneven batch, the discrete adjoint in 3D and 2D, and a training step of the surrogate.

A case is a dict of plain values, ``kind`` among them:

* ``grid``: one plan kept on the device, as a parameter sweep or a design loop keeps it. A pass loads a new material,
  resets the plan, replays its captured steps and reads fields, traces and DFT planes back (``NativeGrid``, as
  ``Simulation.run`` and ``TransmissionProblem.trace`` use it).
* ``batch``: independent 2D TMz grids of uneven sizes advanced together (``NativeBatch``, as ``run_tensor_batch``
  uses it): create the batch, step, release it, read every grid back.
* ``adjoint``: signals (or DFT planes) of a permittivity and the gradient of an objective (``DifferentiableSimulation``,
  ``DifferentiablePlaneSimulation``): forward, replay and reverse steps.
* ``surrogate``: one optimiser step of the convolutional operator on a batch of densities (``ConvNeuralOperator``).

``exact`` steps the same equations in float64 with plain torch operations. The plan's float64 tables (CPML
coefficients, waveforms, monitor corners, incident-line maps) are inputs of the timed calls and of ``exact`` alike.
"""
import math

import numpy as np
import torch

C0 = 299792458.0
L2_BYTES = 126e6


# ---- the listed cases --------------------------------------------------------------------------------------
def listed():
    grid = dict(kind='grid', dim=3, precision='float32', sampling='cell', mesh='uniform', xy='pml', zmax='pml', pml=12,
                source='point', monitor='probe', dispersive=0)
    flat = dict(grid, dim=2, nz=1, pml=16)
    return [
        # The smallest: a TE strip of a photonic-crystal row, periodic across it; every step is launch latency.
        dict(flat, name='te_periodic_200x121', nx=200, ny=121, steps=192, xy='periodic_y', source='te'),
        # A 2D TMz waveguide run at its full length (the plain 2D benchmark scene's size): latency bound, fits on chip.
        dict(flat, name='tmz_320x240', nx=320, ny=240, steps=2000),
        # The batched dataset run: 64 uneven 2D grids, more state than L2 holds.
        dict(kind='batch', name='batch_64_uneven', count=64, lo=128, hi=1024, pml=16, precision='float32', steps=160),
        # A small 3D strip waveguide with a DFT plane: mostly CPML cells, L2 resident.
        dict(grid, name='strip_160x120x40_plane', nx=160, ny=120, nz=40, steps=240, monitor='plane'),
        # A double-precision metasurface unit cell: odd sizes, periodic x and y, per-component permittivity.
        dict(grid, name='unitcell_151x133x117_f64', nx=151, ny=133, nz=117, steps=32, precision='float64', sampling='yee',
             xy='periodic', pml=10),
        # The largest: the 3D benchmark scene, HBM bound.
        dict(grid, name='yee_512x512x256', nx=512, ny=512, nz=256, steps=20),
        # A graded mesh refined around a block (metric factors on every axis).
        dict(grid, name='graded_306x306x176', nx=600, ny=600, nz=320, steps=20, mesh='graded', sampling='yee'),
        # Plane-wave scattering: a total-field / scattered-field box around a scatterer.
        dict(grid, name='tfsf_256', nx=256, ny=256, nz=256, steps=40, source='tfsf'),
        # Metal and dispersive glass: auxiliary differential equations beside the Yee update, odd sizes.
        dict(grid, name='dispersive_201x187x163', nx=201, ny=187, nz=163, steps=24, dispersive=2),
        # Inverse design in 3D: gradient of a mode overlap on a DFT plane through the discrete adjoint.
        dict(kind='adjoint', name='adjoint_200x200x80', dim=3, nx=200, ny=200, nz=80, steps=100, pml=12, precision='float32',
             observe='plane'),
        # Inverse design in 2D: the adjoint step of the transmission design loop.
        dict(kind='adjoint', name='adjoint_tmz_400x400', dim=2, nx=400, ny=400, nz=1, steps=500, pml=16, precision='float32',
             observe='probe'),
        # One optimiser step of the surrogate on the batch size of its benchmark.
        dict(kind='surrogate', name='surrogate_train_256', batch=256, side=100, outputs=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['tmz', 'te', 'batch', 'strip', 'cube', 'cube', 'periodic', 'graded', 'tfsf', 'dispersive', 'adjoint3d',
                       'adjoint2d', 'surrogate'])
    c = dict(kind='grid', dim=3, precision='float32', sampling='cell', mesh='uniform', xy='pml', zmax='pml', pml=rng.randint(6, 16),
             source='point', monitor='probe', dispersive=0)
    if kind in ('tmz', 'te'):
        nx, ny = _log(rng, 64, 1400), _log(rng, 64, 1400)
        c.update(dim=2, nx=nx, ny=ny, nz=1, precision=rng.choice(['float32', 'float32', 'float64']),
                 steps=16 * max(6, min(100, int(4e7 / (nx * ny) / 16))))
        if kind == 'te':
            c.update(source='te', xy=rng.choice(['pml', 'periodic_y']))
        return c
    if kind == 'batch':
        return dict(kind='batch', count=rng.randint(3, 40), lo=rng.randint(64, 200), hi=rng.randint(300, 1000), pml=rng.randint(8, 20),
                    precision=rng.choice(['float32', 'float32', 'float64']), steps=rng.randint(40, 120))
    if kind == 'adjoint3d':
        n = [_log(rng, 48, 180) for _ in range(2)] + [_log(rng, 40, 80)]
        return dict(kind='adjoint', dim=3, nx=n[0], ny=n[1], nz=n[2], steps=rng.randint(40, 90), pml=rng.randint(5, 12),
                    precision=rng.choice(['float32', 'float32', 'float64']), observe=rng.choice(['plane', 'probe']))
    if kind == 'adjoint2d':
        return dict(kind='adjoint', dim=2, nx=_log(rng, 100, 400), ny=_log(rng, 100, 400), nz=1, steps=rng.randint(100, 400), pml=rng.randint(8, 16),
                    precision=rng.choice(['float32', 'float64']), observe='probe')
    if kind == 'surrogate':
        return dict(kind='surrogate', batch=_log(rng, 16, 250), side=rng.randint(30, 100), outputs=rng.choice([16, 32]))
    if kind == 'strip':
        c.update(nx=_log(rng, 60, 200), ny=_log(rng, 60, 160), nz=_log(rng, 40, 60), steps=16 * rng.randint(4, 12), monitor='plane',
                 sampling=rng.choice(['cell', 'yee']))
    elif kind == 'graded':
        c.update(nx=_log(rng, 160, 560), ny=_log(rng, 160, 560), nz=_log(rng, 120, 300), steps=16, mesh='graded', sampling='yee',
                 precision=rng.choice(['float32', 'float32', 'float64']))
    else:
        n = [_log(rng, 60, 420) for _ in range(3)]
        while n[0] * n[1] * n[2] > 3e7:
            n[rng.randrange(3)] //= 2
            n = [max(48, v) for v in n]
        c.update(nx=n[0], ny=n[1], nz=n[2], steps=16 * rng.randint(1, 2), precision=rng.choice(['float32', 'float32', 'float64']))
        if kind == 'cube':
            c.update(zmax=rng.choice(['pml', 'pec']), sampling=rng.choice(['cell', 'yee']))
        elif kind == 'periodic':
            c.update(xy=rng.choice(['periodic', 'periodic_y']), sampling=rng.choice(['cell', 'yee']))
        elif kind == 'tfsf':
            while c['nx'] * c['ny'] * c['nz'] > 1.2e7:
                axis = rng.choice(['nx', 'ny', 'nz'])
                c[axis] = max(48, c[axis] // 2)
            c.update(source='tfsf', pml=rng.randint(6, 10), steps=40)
        else:
            c.update(dispersive=rng.randint(1, 3), pml=rng.randint(6, 10))
    return c


# ---- scenes --------------------------------------------------------------------------------------------------
def _faces(case):
    from torchfdtd_b200 import Boundaries, BoundaryFace
    layers = case['pml']
    pml = BoundaryFace(sigma_scale=3.2 * (layers + 1) / 40, kappa=1, alpha=.05, polynomial=3, alpha_polynomial=1)
    axes = 'xy' if case['dim'] == 2 else 'xyz'
    faces = {f'{a}_{s}': pml for a in axes for s in ('min', 'max')}
    wrap = {'pml': '', 'periodic': 'xy', 'periodic_y': 'y'}[case.get('xy', 'pml')]
    faces.update({f'{a}_{s}': BoundaryFace(kind='periodic') for a in wrap for s in ('min', 'max')})
    if case.get('zmax') == 'pec' and case['dim'] == 3:
        faces['z_max'] = BoundaryFace(kind='pec')
    return Boundaries(**faces)


def _project(case, h=.05):
    """The scene without its permittivity: region, sources and monitors (and the dispersive bodies)."""
    from torchfdtd_b200 import FieldMonitor, Material, Monitor, Project, Region, Source, SpectrumSettings, Structure
    from torchfdtd_b200.models import RunControl
    two_d = case['dim'] == 2
    size = (case['nx'] * h, case['ny'] * h, 1 if two_d else case['nz'] * h)
    extra = {}
    if case.get('mesh') == 'graded':
        extra = dict(mesh_type='graded', mesh_max=3 * h, mesh_grading=1.4, mesh_ppw=6)
    region = Region(dimension='2d' if two_d else '3d', size=size, mesh=h, pml_cells=case['pml'], steps=max(10, case['steps']),
                    precision=case['precision'], material_sampling=case.get('sampling', 'cell'), backend='cuda', cuda_kernel='fused',
                    boundaries=_faces(case), run_control=RunControl(divergence_check=False), snapshot_interval=10000, **extra)
    # A pulse of a few cycles whose peak falls inside the run, so that the fields are alive in every case.
    dt = region.time_step
    peak = min(.4 * case['steps'], 300) * dt
    pulse = dict(wavelength=20 * h * 1.55, pulse='gaussian', time_definition='standard', pulse_length=.6 * peak, pulse_offset=peak)
    component = 'Hz' if case.get('source') == 'te' else 'Ez' if two_d else 'Ey'
    reach = min(6, case['nx'] // 8) * h
    spectrum = SpectrumSettings(sampling='custom', custom_frequencies_hz=[C0 / (20 * h * 1.55e-6)], apodization='none')
    sources = [Source(id='src', center=(-reach, 0, 0), component=component, **pulse)]
    if case.get('source') == 'tfsf':
        inner = tuple((n - 2 * case['pml'] - 16) * h for n in (case['nx'], case['ny'], case['nz']))
        sources = [Source(id='box', kind='tfsf', normal='x', direction='+', size=inner, component='Ey', **pulse)]
    if case.get('monitor') == 'plane' or case.get('observe') == 'plane':
        interior = [(n - 2 * case['pml'] - 4) * h for n in (case['ny'], case['nz'])]
        monitors = [FieldMonitor(id='out', normal='x', center=(reach, 0, 0), size=(0, .6 * interior[0], .6 * interior[1]),
                                 dft_precision='float64', spectrum=spectrum)]
    else:
        monitors = [Monitor(id='probe', center=(reach, 0, 0), component=component, spectrum=spectrum)]
    materials, structures = [], []
    if case.get('mesh') == 'graded':
        materials = [Material(name='Si', index=3.476)]
        structures = [Structure(id='block', size=tuple(.2 * v for v in size), material='Si')]
    if case.get('dispersive'):
        lorentz = dict(resonance_rad_s=3e15, linewidth_rad_s=2e14, delta_epsilon=1.2)
        materials = [Material(name='metal', model='drude', epsilon_inf=1.5, plasma_rad_s=9e15, collision_rad_s=1e14),
                     Material(name='glass', model='lorentz', epsilon_inf=2.0, **lorentz),
                     Material(name='fit', model='multipole', epsilon_inf=1.8,
                              poles=[dict(resonance_rad_s=3e15, strength_rad_s_squared=5e30, damping_rad_s=1e14),
                                     dict(resonance_rad_s=5e15, strength_rad_s_squared=8e30, damping_rad_s=3e14)])]
        r = .12 * min(size)
        structures = [Structure(id='ball', kind='sphere', center=(3 * r, 0, 0), radius=r, material='metal'),
                      Structure(id='slab', size=(r, .8 * size[1], .8 * size[2]), center=(-2 * r, 0, 0), material='glass'),
                      Structure(id='rod', size=(r, r, .5 * size[2]), center=(0, 2 * r, 0), material='fit')][:case['dispersive']]
    own = dict(materials=materials, structures=structures) if materials else {}
    return Project(region=region, sources=sources, monitors=monitors, **own)


def _generator(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _blocks(shape, seed, lo, hi, dtype, edge=8):
    """A piecewise-constant permittivity: uniform in [lo, hi] on blocks of 8 cells per side."""
    small = [(n + edge - 1) // edge for n in shape]
    v = torch.rand(small, generator=_generator(seed), device='cuda', dtype=torch.float64) * (hi - lo) + lo
    for axis, n in enumerate(shape):
        v = v.repeat_interleave(min(edge, n), dim=axis).narrow(axis, 0, n)
    return v.to(dtype).contiguous()


def _grid_plan(case, seed):
    """(plan, relative permittivity on the device): what a program has before it steps a plan."""
    from torchfdtd_b200.plan import plan_grid
    project = _project(case)
    dtype = torch.float64 if case['precision'] == 'float64' else torch.float32
    plan = plan_grid(project, material=bool(case.get('dispersive')))
    eps = _blocks(plan.shape, seed, 1, 12.1, dtype)
    if case.get('dispersive'):
        keep = torch.as_tensor(np.asarray(plan.epsilon), device='cuda').to(dtype)
        owned = torch.zeros(eps.numel() * 3, dtype=torch.bool, device='cuda')
        for st in plan.ade:
            owned[torch.as_tensor(st.target, device='cuda')] = True
        eps = torch.where(owned.view(*plan.shape, 3).any(-1), keep, 1 + (eps - 1) * .25)
    if case.get('source') == 'tfsf':
        # The scatterer fills the box up to four cells from its faces, which stand in the background.
        inside = torch.zeros(plan.shape, dtype=torch.bool, device='cuda')
        inset = case['pml'] + 12
        inside[tuple(slice(inset, n - inset) for n in plan.shape)] = True
        eps = torch.where(inside, eps, torch.ones_like(eps))
    if case.get('sampling') == 'yee':
        eps = torch.stack([eps, eps.roll(1, 0), eps.roll(1, 1)], dim=-1)
    plan.epsilon, plan.inv_eps = eps, (plan.inv_eps if case.get('dispersive') else None)
    return plan, eps


def _batch_sides(case, seed):
    """Sides of the batch's grids: fixed by the case, so that every seed does the same work."""
    rng = np.random.default_rng(2024 + case['count'])
    return [tuple(int(v) for v in s) for s in rng.integers(case['lo'], case['hi'] + 1, size=(case['count'], 2))]


def _batch_members(case, seed):
    out = []
    for k, (nx, ny) in enumerate(_batch_sides(case, seed)):
        member = dict(kind='grid', dim=2, nx=nx, ny=ny, nz=1, steps=case['steps'], pml=case['pml'], precision=case['precision'])
        out.append(_grid_plan(member, seed * 1000 + k))
    return out


def _adjoint_scene(case, seed):
    from torchfdtd_b200.adjoint import DifferentiablePlaneSimulation, DifferentiableSimulation
    project = _project(case, h=.04)
    model = (DifferentiablePlaneSimulation if case['observe'] == 'plane' else DifferentiableSimulation)(project)
    dtype = torch.float64 if case['precision'] == 'float64' else torch.float32
    # A density smoothed over a few cells in the middle of an oxide background.
    shape = model.plan.shape
    rho = _blocks(shape, seed, 0, 1, torch.float64, edge=4)
    inside = torch.zeros(shape, dtype=torch.float64, device='cuda')
    inside[tuple(slice(n // 3, n - n // 3) if n > 1 else slice(None) for n in shape)] = 1
    eps = (2.085 + rho * inside * (12.08 - 2.085)).to(dtype)
    return model, eps


def _weights(seed, *shape):
    return torch.randn(shape, generator=_generator(seed + 77), device='cuda', dtype=torch.float64)


def _surrogate_inputs(case, seed):
    n, s = case['batch'], case['side']
    noise = torch.randn((n, 1, s, s), generator=_generator(seed), device='cuda')
    smooth = torch.nn.functional.avg_pool2d(noise, 7, stride=1, padding=3)
    rho = torch.sigmoid(4 * smooth / smooth.std())[:, 0].contiguous()
    target = .5 * torch.randn((n, case['outputs']), generator=_generator(seed + 1), device='cuda')
    return rho, target


# ---- prepare and run -----------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case['kind']
    if kind == 'grid':
        from torchfdtd_b200.native import NativeGrid
        plan, eps = _grid_plan(case, seed)
        inv = (1 / eps).contiguous()
        grid = NativeGrid(plan, material=inv)
        # The captured steps a program replays: 20 or 16 steps to a graph where they divide the run.
        width = next(w for w in (20, 16, 8, 4, 2, 1) if case['steps'] % w == 0)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            grid.step(1, stream)
            grid.reset()
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            graph.capture_begin()
            grid.step(width, stream)
            graph.capture_end()
        torch.cuda.synchronize()
        return dict(kind=kind, grid=grid, inv=inv, graph=graph, replays=case['steps'] // width, planes=len(plan.planes))
    if kind == 'batch':
        from torchfdtd_b200.native import NativeGrid
        members = _batch_members(case, seed)
        grids = [NativeGrid(plan, kernel='tile2d', material=(1 / eps).contiguous()) for plan, eps in members]
        return dict(kind=kind, grids=grids, steps=case['steps'])
    if kind == 'adjoint':
        model, eps = _adjoint_scene(case, seed)
        model.engine(eps)
        return dict(kind=kind, model=model, eps=eps, observe=case['observe'], seed=seed, steps=case['steps'])
    from torchfdtd_b200.surrogate import ConvNeuralOperator
    rho, target = _surrogate_inputs(case, seed)
    net = ConvNeuralOperator(outputs=case['outputs'], seed=seed, input_shape=(case['side'], case['side']))
    return dict(kind=kind, net=net, rho=rho, target=target)


def _mode(points, like):
    """A Gaussian mode profile over the plane's points."""
    return torch.exp(-torch.linspace(-1, 1, points, device='cuda', dtype=torch.float64) ** 2).to(like.dtype)


def run(state):
    kind = state['kind']
    if kind == 'grid':
        grid = state['grid']
        grid.set_material(state['inv'])
        grid.reset()
        for _ in range(state['replays']):
            state['graph'].replay()
        E, H = grid.fields_device()
        return dict(E=E, H=H, traces=grid.traces_device(), planes=[grid.get_plane(k) for k in range(state['planes'])])
    if kind == 'batch':
        from torchfdtd_b200.native import NativeBatch
        grids = state['grids']
        for g in grids:
            g.reset()
        batch = NativeBatch(grids)
        batch.step(state['steps'])
        batch.close()
        fields = [g.fields_device() for g in grids]
        return dict(E=torch.cat([e.reshape(-1) for e, _ in fields]), H=torch.cat([h.reshape(-1) for _, h in fields]),
                    traces=torch.cat([g.traces_device() for g in grids], dim=1))
    if kind == 'adjoint':
        eps = state['eps'].detach().requires_grad_(True)
        if state['observe'] == 'plane':
            seen = state['model'](eps)['out'].fields
            ey = seen[..., 1]
            objective = (torch.abs((ey * _mode(ey.shape[1], ey)).sum(dim=1)) ** 2).sum() / abs(ey.detach()).max() ** 2
        else:
            seen = state['model'](eps).signals
            objective = (seen * _weights(state['seed'], *seen.shape).to(seen.dtype)).sum()
        gradient, = torch.autograd.grad(objective, eps)
        return dict(seen=seen.detach(), gradient=gradient)
    net = state['net']
    out_before = net.train_step(state['rho'], state['target'])
    return dict(loss=out_before, gradients={k: v.clone() for k, v in net.grads.items()})


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _step_work(nx, ny, nz, case, comps, samples):
    """(bytes, flops, state bytes) of one time step: each advanced component read and written, the permittivity read,
    the CPML memories read and written; two differences, their sum and the update per component."""
    real = 8 if case['precision'] == 'float64' else 4
    cells = nx * ny * nz
    wrap = {'pml': (), 'periodic': (0, 1), 'periodic_y': (1,)}[case.get('xy', 'pml')]
    n, L = (nx, ny, nz), case['pml']
    psi = sum(2 * L * cells // n[a] * (4 if comps == 6 else 2) for a in range(3) if n[a] > 1 and a not in wrap)
    moved = real * (cells * (2 * comps + samples) + 2 * psi)
    return moved, cells * comps * 5.5, real * (cells * (comps + samples) + psi)


def work(case):
    kind, steps = case['kind'], case.get('steps', 1)
    if kind in ('grid', 'adjoint'):
        # A graded mesh keeps about half the cells per axis of its base lattice.
        shape = [n // 2 if case.get('mesh') == 'graded' and n > 1 else n for n in (case['nx'], case['ny'], case['nz'])]
        comps = 6 if case['dim'] == 3 else 3
        samples = 3 if case.get('sampling') == 'yee' and comps == 6 else 1
        moved, flops, held = _step_work(*shape, case, comps, samples)
        cells = shape[0] * shape[1] * shape[2]
        real = 8 if case['precision'] == 'float64' else 4
        ends = real * cells * (6 + samples)                       # the material in, the fields out
        if kind == 'grid':
            # State that L2 holds needs no HBM traffic between the steps.
            return dict(bytes=ends + (steps * moved if held > L2_BYTES else 2 * held), flops=steps * flops)
        # Forward, one recomputation and the transpose (the adjoint fields and the sensitivity read and written).
        reverse = moved + real * cells * (3 * 2 + comps)
        both = held + real * cells * (3 * 2 + comps // 2)
        return dict(bytes=real * cells * 2 + (steps * (2 * moved + reverse) if both > L2_BYTES else 2 * held + both), flops=4 * steps * flops)
    if kind == 'batch':
        total = [_step_work(nx, ny, 1, case, 3, 1) for nx, ny in _batch_sides(case, 0)]
        moved, flops, held = (sum(t[i] for t in total) for i in range(3))
        ends = (8 if case['precision'] == 'float64' else 4) * sum(6 * a * b for a, b in _batch_sides(case, 0))
        return dict(bytes=ends + (steps * moved if held > L2_BYTES else 2 * held), flops=steps * flops)
    n, s = case['batch'], case['side']
    moved, flops, ci = n * s * s * 4, 0, 4
    for stride in (1, 2, 1, 2, 1, 2, 1, 2):
        s = (s - 1) // stride + 1
        flops += 3 * 2 * n * s * s * 64 * 9 * ci                  # forward, backward data, backward weight
        moved += 2 * 64 * n * s * s * 8                           # z and a written, a read twice, dz written and read twice, z read
        ci = 64
    weights = 64 * 9 * (16 + 7 * 64) + case['outputs'] * s * s * 64
    return dict(bytes=moved + 4 * 7 * weights, flops=flops)


def tolerance(case):
    if case['kind'] == 'surrogate':
        return {'rel': 2e-2, 'max': .6}
    if case['precision'] == 'float64':
        return {'rel': 1e-13, 'max': 1e-11}
    return {'rel': 3e-5, 'max': 3e-3}


# ---- float64 -------------------------------------------------------------------------------------------------
# (derivative axis, input component, output component, sign) of a curl.
TERMS = ((0, 2, 1, -1), (0, 1, 2, 1), (1, 2, 0, 1), (1, 0, 2, -1), (2, 1, 0, -1), (2, 0, 1, 1))


class _Exact:
    """The Yee / CPML time loop of a plan in float64 torch operations (differentiable in the inverse permittivity)."""

    def __init__(self, plan, inv, active=range(6)):
        f = dict(device='cuda', dtype=torch.float64)
        self.plan, self.active = plan, set(active)
        self.inv = [inv[..., c] for c in range(3)] if inv.ndim == 4 else [inv] * 3
        self.F = [[torch.zeros(plan.shape, **f) for _ in range(3)] for _ in range(2)]
        self.psi = {}
        self.slabs, self.metric = {}, {}
        for forward in (False, True):
            for axis in range(3):
                view = [1, 1, 1]
                view[axis] = -1
                self.slabs[forward, axis] = sorted(
                    ((s.lo, s.hi, *(torch.as_tensor(v, **f).view(view) for v in (s.b, s.c, s.inv_kappa)))
                     for s in plan.segments if s.forward == forward and s.axis == axis), key=lambda s: s[0])
                if (forward, axis) in plan.metrics:
                    values, wrap = plan.metrics[forward, axis]
                    self.metric[forward, axis] = (torch.as_tensor(values, **f).view(view), wrap)
        self.lines = [dict(box=b, e=torch.zeros(b.count, **f), h=torch.zeros(b.count, **f), pe=torch.zeros(b.count, **f),
                           ph=torch.zeros(b.count, **f), coef=[[torch.as_tensor(v, **f) for v in p] for p in b.coefficients],
                           maps={k: [torch.as_tensor(v, device='cuda') for v in m] for k, m in b.maps.items()}) for b in plan.tfsf]
        self.ade = []
        for st in plan.ade:
            target = torch.as_tensor(st.target, device='cuda')
            for c in range(3):
                cell = target[target % 3 == c] // 3
                if cell.numel():
                    pole = [torch.as_tensor(v, **f).view(-1, 1) for v in (st.a, st.d, st.k)]
                    zero = torch.zeros((st.poles, cell.numel()), **f)
                    self.ade.append(dict(c=c, cell=cell, eps=st.eps_inf, pole=pole, P=zero, Q=zero.clone()))

    def curl(self, family):
        forward, plan = family == 1, self.plan
        src = self.F[1 - family]
        out = [None, None, None]
        for axis, comp, o, sign in TERMS:
            n = plan.shape[axis]
            if n == 1 or 3 * family + o not in self.active:
                continue
            field = src[comp]
            d = torch.diff(field, dim=axis)
            if (forward, axis) in self.metric:
                d = d * self.metric[forward, axis][0]
            start, parts, at = 0 if forward else 1, [], 0
            for k, (lo, hi, b, c, inv_k) in enumerate(self.slabs[forward, axis]):
                lo, hi, key = lo - start, hi - start, (family, axis, o, k)
                part = d.narrow(axis, lo, hi - lo)
                memory = c * part + (b * self.psi[key] if key in self.psi else 0)
                self.psi[key] = memory
                parts += [d.narrow(axis, at, lo - at), part * inv_k + memory]
                at = hi
            d = torch.cat([*parts, d.narrow(axis, at, n - 1 - at)], dim=axis)
            first, last = field.narrow(axis, 0, 1), field.narrow(axis, n - 1, 1)
            if plan.faces[axis][0] == 'periodic':
                edge = (first - last) * (self.metric[forward, axis][1] if (forward, axis) in self.metric else 1)
            elif forward and axis in plan.pec_upper:
                edge = -plan.pec_upper[axis] * last
            else:
                edge = torch.zeros_like(first)
            d = torch.cat([d, edge] if forward else [edge, d], dim=axis)
            out[o] = sign * d if out[o] is None else out[o] + sign * d
        return out

    def step(self, n):
        plan = self.plan
        for family in range(2):
            old = [self.F[family][m['c']].view(-1)[m['cell']] for m in self.ade] if family == 0 else []
            for c, curl in enumerate(self.curl(family)):
                if curl is not None:
                    scale = plan.courant * self.inv[c] if family == 0 else -plan.courant
                    self.F[family][c] = self.F[family][c] + scale * curl
            for m, was in zip(self.ade, old):
                a, d, k = m['pole']
                response = (m['Q'] - a * m['P']) / d
                flat = self.F[0][m['c']].view(-1)
                new = (m['eps'] * flat[m['cell']] - k.sum() * was - response.sum(0)) / (m['eps'] + k.sum())
                delta = response + k * (new + was)
                m['P'], m['Q'] = m['P'] + delta, 2 * delta - m['Q']
                flat[m['cell']] = new
            for t in plan.sources:
                if t.family == family:
                    field = self.F[family][t.comp].clone()
                    field[tuple(slice(lo, hi) for lo, hi in zip(t.lo, t.hi))] += float(t.values[n])
                    self.F[family][t.comp] = field
            for line in self.lines:
                self.incident(line, family, n)

    def incident(self, line, family, n):
        box, e, h = line['box'], line['e'], line['h']
        zero = e.new_zeros(1)
        diff = torch.cat([torch.diff(e), zero]) if family else torch.cat([zero, torch.diff(h)])
        b, c = line['coef'][family]
        name, memory = ('h', 'ph') if family else ('e', 'pe')
        line[memory] = line[memory] * b + c * diff
        line[name] = line[name] - (box.courant if family else box.courant_e) * (diff + line[memory])
        if family == 0:
            line['e'][box.drive_at] += float(box.drive[n])
        target, sample, weight = line['maps']['H' if family else 'E']
        incident = (line['e'] if family else h)[sample] * weight
        for k in range(3):
            mine = target % 3 == k
            self.F[family][k].view(-1).index_add_(0, target[mine] // 3, incident[mine])

    def value(self, name):
        return self.F[0 if name[0] == 'E' else 1]['xyz'.index(name[1].lower())]

    def run(self, steps, cells=None):
        """Steps, with the traces of the plan (or the values at ``cells``: pairs of component and cell) of each."""
        plan = self.plan
        wanted = [(t.component, t.index) for t in plan.traces] if cells is None else cells
        groups = {}
        for k, (name, cell) in enumerate(wanted):
            groups.setdefault(name, []).append((k, cell))
        order = torch.as_tensor([k for g in groups.values() for k, _ in g], device='cuda', dtype=torch.long)
        where = {name: [torch.as_tensor(v, device='cuda') for v in zip(*(c for _, c in g))] for name, g in groups.items()}
        planes = [dict(p=p, cell=torch.as_tensor(p.corner_cells, device='cuda'),
                       weight=torch.as_tensor(p.corner_weights, device='cuda').double(),
                       sum=torch.zeros((len(p.frequency), p.corner_cells.shape[2], len(p.components)), device='cuda',
                                       dtype=torch.complex128)) for p in plan.planes] if cells is None else []
        rows = []
        for n in range(steps):
            self.step(n)
            rows.append(torch.cat([self.value(name)[tuple(ix)] for name, ix in where.items()])
                        if wanted else self.F[0][0].new_zeros(0))
            for q in planes:
                p = q['p']
                for k, name in enumerate(p.components):
                    late = name[0] == 'H'
                    sample = (self.value(name).reshape(-1)[q['cell'][k]] * q['weight'][k]).sum(0) * float(p.windows[int(late)][n])
                    phase = np.exp(2j * np.pi * p.frequency * plan.time_step * (n + 1 + .5 * late))
                    q['sum'][..., k] += torch.as_tensor(phase, device='cuda')[:, None] * sample[None]
        seen = torch.stack(rows)
        return torch.zeros_like(seen).index_copy(1, order, seen) if wanted else seen, [q['sum'] for q in planes]

    def fields(self, family):
        return torch.stack(self.F[family], dim=-1)


def _active(plan):
    return [['Ex', 'Ey', 'Ez', 'Hx', 'Hy', 'Hz'].index(c) for c in plan.active_components()]


def _exact_adjoint(case, seed):
    model, eps = _adjoint_scene(case, seed)
    plan = model.plan
    eps = eps.double().requires_grad_(True)
    loop = _Exact(plan, 1 / eps, _active(plan))
    samples, _ = loop.run(case['steps'], [(t.component, t.index) for t in plan.traces])
    if case['observe'] == 'probe':
        seen = samples
        objective = (seen * _weights(seed, *seen.shape)).sum()
    else:
        from torchfdtd_b200.plan import plan_grid
        p, = plan_grid(model.project, material=False).planes
        column = {(t.component, tuple(int(v) for v in t.index)): k for k, t in enumerate(plan.traces)}
        fields = []
        for k, name in enumerate(p.components):
            cells = np.stack(np.unravel_index(p.corner_cells[k], plan.shape), axis=-1)
            at = torch.as_tensor([[column[name, tuple(int(v) for v in c)] for c in row] for row in cells], device='cuda')
            times = (np.arange(case['steps']) + 1 + (.5 if name[0] == 'H' else 0)) * plan.time_step
            kernel = torch.as_tensor(np.exp(2j * np.pi * p.frequency[:, None] * times) * plan.time_step, device='cuda')
            values = (samples[:, at] * torch.as_tensor(p.corner_weights[k], device='cuda').double()).sum(1)
            fields.append(kernel @ values.to(kernel.dtype))
        by_name = dict(zip(p.components, fields))
        seen = torch.stack([by_name.get(c, torch.zeros_like(fields[0])) for c in ('Ex', 'Ey', 'Ez', 'Hx', 'Hy', 'Hz')], dim=-1)
        ey = seen[..., 1]
        objective = (torch.abs((ey * _mode(ey.shape[1], ey)).sum(dim=1)) ** 2).sum() / abs(ey.detach()).max() ** 2
    gradient, = torch.autograd.grad(objective, eps)
    return dict(seen=seen.detach(), gradient=gradient)


def _exact_surrogate(case, seed):
    """The network, its loss and every gradient in float64 (no bfloat16 rounding anywhere)."""
    rho, target = _surrogate_inputs(case, seed)
    n, s, layers = case['batch'], case['side'], ((16, 1), (64, 2), (64, 1), (64, 2), (64, 1), (64, 2), (64, 1), (64, 2))
    g = torch.Generator(device='cpu').manual_seed(seed)
    params = {}
    for k, (ci, _) in enumerate(layers):
        params[f'w{k}'] = torch.randn((9, 64, ci), generator=g) * math.sqrt(2 / (9 * (4 if k == 0 else ci)))
        params[f'b{k}'] = torch.zeros(64)
    side = s
    for _, stride in layers:
        side = (side - 1) // stride + 1
    params['wh'] = torch.randn((case['outputs'], side * side * 64), generator=g) / math.sqrt(side * side * 64)
    params['bh'] = torch.zeros(case['outputs'])
    params = {k: v.cuda().double().requires_grad_(True) for k, v in params.items()}
    axis = torch.linspace(-1, 1, s, device='cuda', dtype=torch.float64)
    x = torch.zeros((n, 16, s, s), device='cuda', dtype=torch.float64)
    x[:, 0], x[:, 1], x[:, 2], x[:, 3] = 2 * rho.double() - 1, axis[None, None, :], axis[None, :, None], 1
    for k, (ci, stride) in enumerate(layers):
        w = params[f'w{k}'].view(3, 3, 64, ci).permute(2, 3, 0, 1)
        with torch.backends.cudnn.flags(enabled=False):
            z = torch.nn.functional.conv2d(x, w, params[f'b{k}'], stride=stride, padding=1)
        x = torch.nn.functional.gelu(z, approximate='tanh')
    out = x.permute(0, 2, 3, 1).reshape(n, -1) @ params['wh'].T + params['bh']
    loss = ((out - target.double()) ** 2).mean()
    grads = torch.autograd.grad(loss, list(params.values()))
    return dict(loss=loss.detach().reshape(1), gradients=dict(zip(params, grads)))


def exact(case, seed):
    kind = case['kind']
    if kind == 'surrogate':
        return _exact_surrogate(case, seed)
    if kind == 'adjoint':
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        if kind == 'grid':
            plan, eps = _grid_plan(case, seed)
            loop = _Exact(plan, 1 / eps.double(), _active(plan))
            seen, planes = loop.run(case['steps'])
            return dict(E=loop.fields(0), H=loop.fields(1), traces=seen, planes=planes)
        E, H, traces = [], [], []
        for plan, eps in _batch_members(case, seed):
            loop = _Exact(plan, 1 / eps.double(), _active(plan))
            traces.append(loop.run(case['steps'])[0])
            E.append(loop.fields(0).reshape(-1))
            H.append(loop.fields(1).reshape(-1))
        return dict(E=torch.cat(E), H=torch.cat(H), traces=torch.cat(traces, dim=1))

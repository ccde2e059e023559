"""The task list and the plan's own numbering at their edges, against the CPU
oracle (every J/K element within 1e-10, as the parity tests): one quartet
shared by a warp's lanes, shells in an order unlike the plan's, and classes
of more rows than one scan tile."""
import numpy as np
import pytest

from electrolites_b200 import clusters
from electrolites_b200.gto import Mole

pytestmark = pytest.mark.gpu

ATOL = 1e-10
TOL = 1e-13


@pytest.fixture(scope='module')
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    return torch


def _check(torch, oracle, mol, dms, hermi):
    from electrolites_b200.jk import VHFOpt
    opt = VHFOpt(mol, TOL).build()
    vj, vk = opt.get_jk(torch.as_tensor(dms), hermi)
    rj, rk, _ = oracle.jk(mol, dms, tol=TOL)
    assert float(np.abs(vj.cpu().numpy() - rj).max()) <= ATOL
    assert float(np.abs(vk.cpu().numpy() - rk).max()) <= ATOL


@pytest.mark.parametrize('nprim', [1, 2, 3, 5, 6, 7, 11, 12, 19])
@pytest.mark.parametrize('l', [0, 1])
def test_one_shell_of_many_primitives(torch, oracle, nprim, l):
    """A single shell: one quartet, whose nprim^4 primitive quartets the lanes
    of a warp share in parts that need not divide them; from 12 primitives on
    the plan splits its pair (more than 128 primitive pairs)."""
    prims = [(0.2 * 1.6 ** k, 1.0 / (k + 1)) for k in range(nprim)]
    mol = Mole([('H', (0.1, -0.2, 0.3))], basis={'H': [[l] + prims]}, cart=True)
    n = mol.nao_cart
    d = np.random.default_rng(nprim).standard_normal((2, n, n))
    _check(torch, oracle, mol, d + d.transpose(0, 2, 1), 1)


@pytest.mark.parametrize('hermi', [1, 0])
@pytest.mark.parametrize('seed', [1, 2])
def test_shells_in_any_order(torch, oracle, hermi, seed):
    """The plan numbers shells by l, kind and place; the caller's order,
    shuffled here across atoms and kinds, is what goes in and comes out."""
    basis = {'O': [[0, (5.0, 0.4), (1.1, 0.7)], [1, (1.3, 0.5), (0.4, 0.6)], [2, (0.8, 1.0)],
                   [0, (0.3, 1.0)], [3, (1.1, 1.0)]],
             'H': [[1, (0.9, 1.0)], [0, (1.2, 0.5), (0.3, 0.6)], [0, (0.15, 1.0)]]}
    mol = Mole(clusters.water_cluster(2, 4.0, seed), basis=basis, cart=True)
    rng = np.random.default_rng(seed)
    mol._bas = mol._bas[rng.permutation(len(mol._bas))]
    n = mol.nao_cart
    d = 0.1 * rng.standard_normal((3, n, n))
    if hermi:
        d = d + d.transpose(0, 2, 1)
    _check(torch, oracle, mol, d, hermi)


def test_rows_of_several_tiles(torch):
    """(H2O)_14: 4851 (ss| rows, five scan tiles; a batch that gives the class
    rows of two molecules.  Builds with one task per row and with few large
    tasks agree (the same quartets in another order)."""
    from electrolites_b200.batch import JKBatch
    from electrolites_b200.jk import VHFOpt, class_keys
    mols = [clusters.water_mole(n, 3.3 * n ** (1 / 3), 5 + n) for n in (14, 3)]
    opts = [VHFOpt(m, TOL).build() for m in mols]
    dms = [torch.as_tensor(clusters.uhf_pair(clusters.atomic_density(m, 3), 4), device='cuda')
           for m in mols]
    ref = [o.get_jk(d, 1) for o, d in zip(opts, dms)]
    counts = [o.class_counts() for o in opts]
    for tasks in (1, 4096):
        for o in opts:
            for c in range(len(class_keys())):
                o.set_tuning(c, tasks)
        for o, d, (rj, rk), n in zip(opts, dms, ref, counts):
            vj, vk = o.get_jk(d, 1)
            assert float((vj - rj).abs().max()) <= ATOL and float((vk - rk).abs().max()) <= ATOL
            assert o.class_counts() == n
    batch = JKBatch()
    vj, vk = batch.build(opts, dms, 1)
    for a, b, (rj, rk) in zip(vj, vk, ref):
        assert float((a - rj).abs().max()) <= ATOL and float((b - rk).abs().max()) <= ATOL


def test_repeated_builds_of_changing_kinds(torch):
    """A small plan's repeated builds replay a graph from the third on: new
    densities and outputs at other addresses, another kind of build in between,
    a loosened and restored threshold, and the J engine off and on again give
    what a fresh plan's first build gives."""
    from electrolites_b200.jk import VHFOpt
    mol = clusters.water_mole(2, 4.2, 17)
    opt = VHFOpt(mol, TOL).build()
    base = clusters.atomic_density(mol, 3)
    rng = np.random.default_rng(5)

    def once(o, k, d):
        if k == 'grad':
            return (o.jk_energy_per_atom(d, 1.0, 0.3),)
        if k == 'rsh':
            return (o.get_k(d, omega=0.4, lr_factor=1.0, sr_factor=0.2),)
        return o.get_jk(d, 0 if k == 'general' else 1, with_k=k != 'j')

    kept = []
    for k in ['jk'] * 5 + ['j'] * 4 + ['jk', 'general'] * 4 + ['grad'] * 4 + ['rsh'] * 4 + ['jk'] * 4:
        p = 1e-2 * rng.standard_normal((2,) + base.shape)
        d = torch.as_tensor(base + (p if k == 'general' else p + p.transpose(0, 2, 1)), device='cuda')
        kept.append(d)                       # every density at an address of its own
        if len(kept) % 7 == 3:
            opt.direct_scf_tol = 1e-8
            once(opt, k, d)
            opt.direct_scf_tol = TOL
        if len(kept) % 5 == 4:
            opt.set_jengine(False)
            once(opt, k, d)
            opt.set_jengine(True)
        got = once(opt, k, d)
        ref = once(VHFOpt(mol, TOL).build(), k, d)
        kept.append(got)
        for a, b in zip(got, ref):
            assert (a is None) == (b is None)
            if a is not None:
                assert float((a - b).abs().max()) <= ATOL


def _once(o, k, d):
    """One call of kind k: the plan's outputs that there are."""
    if k == 'grad':
        return (o.jk_energy_per_atom(d, 1.0, 0.3),)
    if k == 'rsh':
        return (o.get_k(d, omega=0.4, lr_factor=1.0, sr_factor=0.2),)
    if k == 'j':
        return (o.get_j(d),)
    return o.get_jk(d, 0 if k == 'general' else 1)


@pytest.mark.parametrize('kind', ['jk', 'j', 'general', 'grad', 'rsh'])
def test_graph_replay_with_moving_densities(torch, kind):
    """The third build of a kind captures, the later ones replay, with every
    density at an address of its own; two streams in turn share the graph.
    A replay gives what a fresh plan's direct launches give."""
    from electrolites_b200.jk import VHFOpt
    mol = clusters.water_mole(2, 4.2, 17)
    opt = VHFOpt(mol, TOL).build()
    base = clusters.atomic_density(mol, 3)
    rng = np.random.default_rng(6)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    kept = []
    for n in range(8):
        p = 1e-2 * rng.standard_normal((1,) + base.shape)
        d = torch.as_tensor(base + (p if kind == 'general' else p + p.transpose(0, 2, 1)), device='cuda')
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[n % 2]):
            got = _once(opt, kind, d)
        assert opt.stats() == {'graph_replayed': n > 2, 'graph_captured': n == 2}
        kept.append((d, got))
        fresh = VHFOpt(mol, TOL).build()
        for a, b in zip(got, _once(fresh, kind, d)):
            assert float((a - b).abs().max()) <= ATOL
        assert not any(fresh.stats().values())


def test_build_in_the_callers_graph(torch):
    """A build captured into the caller's own graph: its replays give the J/K of
    the densities then in the buffers, jk_sync waits for them, and the plan's
    ordinary builds go on."""
    from electrolites_b200.jk import VHFOpt
    mol = clusters.water_mole(2, 4.2, 17)
    opt = VHFOpt(mol, TOL).build()
    base = torch.as_tensor(clusters.atomic_density(mol, 3)[None], device='cuda')
    dm, vj, vk = base.clone(), torch.empty_like(base), torch.empty_like(base)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(2):                   # warm: buffers, descriptors, kernel attributes
        opt.build_jk_async(dm, 1, vj=vj, vk=vk, stream=st)
    opt.sync(st)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        opt.build_jk_async(dm, 1, vj=vj, vk=vk, stream=st)
    for f in (1.0, 0.7):
        dm.copy_(f * base)
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            g.replay()
        opt.sync(st)
        rj, rk = VHFOpt(mol, TOL).build().get_jk(dm, 1)
        assert float((vj - rj).abs().max()) <= ATOL and float((vk - rk).abs().max()) <= ATOL
    aj, ak = opt.get_jk(base, 1)
    assert float((0.7 * aj - rj).abs().max()) <= ATOL and float((0.7 * ak - rk).abs().max()) <= ATOL
    del g


def test_plans_hold_no_streams(torch):
    """A plan takes its tables and little more of the device (a stream takes
    half a megabyte): 64 plans of one water, built in a batch and each alone,
    stay below a megabyte each."""
    from electrolites_b200.batch import JKBatch
    from electrolites_b200.jk import VHFOpt
    mol = clusters.water_mole(1, 3.0, 7)
    d = torch.as_tensor(clusters.atomic_density(mol, 3)[None], device='cuda')
    batch = JKBatch()
    first = VHFOpt(mol, TOL).build()
    out = [torch.empty((64,) + d.shape, dtype=d.dtype, device='cuda') for _ in range(2)]
    batch.build([first], [d], 1)
    vj, vk = first.get_jk(d, 1)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    opts = [VHFOpt(mol, TOL).build() for _ in range(64)]
    batch.build(opts, [d] * 64, 1, vj=list(out[0]), vk=list(out[1]))
    for o in opts:
        o.build_jk_async(d, 1, vj=vj, vk=vk)
        o.sync()
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
    assert float((out[1][63] - vk).abs().max()) <= ATOL


def test_builds_of_many_streams_and_threads(torch):
    """More streams than the device has sets of side streams, from four threads
    at a time, each plan on its own stream: every build is its plan's."""
    import threading

    from electrolites_b200.jk import VHFOpt
    work = []
    for k in range(12):
        mol = clusters.water_mole(1 + k % 3, 4.5, 40 + k)
        d = torch.as_tensor(clusters.atomic_density(mol, k)[None], device='cuda')
        work.append((VHFOpt(mol, TOL).build(), d, VHFOpt(mol, TOL).build().get_jk(d, 1), torch.cuda.Stream()))
    torch.cuda.synchronize()
    bad = []

    def some(mine):
        for _ in range(6):               # direct builds, a capture, replays
            got = []
            for opt, d, _, st in mine:
                vj, vk = torch.empty_like(d), torch.empty_like(d)
                opt.build_jk_async(d, 1, vj=vj, vk=vk, stream=st)
                got.append((vj, vk))
            for (opt, _, ref, st), g in zip(mine, got):
                opt.sync(st)
                bad.extend(float((a - b).abs().max()) for a, b in zip(g, ref)
                           if not float((a - b).abs().max()) <= ATOL)

    threads = [threading.Thread(target=some, args=(work[k::4],)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def _split_mol():
    """s and d shells of twelve primitives: their pairs have 144 primitive
    pairs and the plan splits them; a second atom of ordinary shells."""
    prims = [(0.15 * 1.7 ** k, 1.0 / (k + 1)) for k in range(12)]
    basis = {'H': [[0] + prims, [2] + prims], 'He': [[0, (0.9, 0.5), (0.3, 0.5)], [1, (0.7, 1.0)]]}
    return Mole([('H', (0.0, 0.1, -0.2)), ('He', (0.8, -0.5, 0.9))], basis=basis, cart=True)


def test_split_pairs_in_every_build(torch, oracle):
    """J/K with symmetric and general densities, J alone by the J engine, the
    (ij|kl) digest and the McMurchie-Davidson kernels (which leave classes of so
    many primitives to the J engine), a batch, a mixed build, an allocation-free
    build and a gradient, all with pairs that the plan splits."""
    import ctypes

    from electrolites_b200 import _lib
    from electrolites_b200.batch import JKBatch
    from electrolites_b200.jk import VHFOpt
    mol = _split_mol()
    n = mol.nao_cart
    rng = np.random.default_rng(8)
    gen = 0.3 * rng.standard_normal((2, n, n))
    dms = gen + gen.transpose(0, 2, 1)
    _check(torch, oracle, mol, dms, 1)
    _check(torch, oracle, mol, gen, 0)
    rj, rk, _ = oracle.jk(mol, dms, tol=TOL)
    opt = VHFOpt(mol, TOL).build()
    d = torch.as_tensor(dms, device='cuda')

    def same(v, ref):
        assert float(np.abs(v.cpu().numpy() - ref).max()) <= ATOL

    same(opt.get_j(d), rj)
    opt.set_jmd(1)
    same(opt.get_j(d), rj)
    opt.set_jmd(-1)
    opt.set_jengine(False)
    same(opt.get_j(d), rj)
    opt.set_jengine(True)
    water = VHFOpt(clusters.water_mole(1, 3.0, 7), TOL).build()
    wd = torch.as_tensor(clusters.atomic_density(water.mol, 3)[None], device='cuda')
    vj, vk = JKBatch().build([water, opt], [wd, d], 1)
    same(vj[1], rj)
    same(vk[1], rk)
    mj, mk = (v.cpu().numpy() for v in opt.get_jk(d, 1, mixed_threshold=1e-6))
    for m, r in ((mj, rj), (mk, rk)):
        assert abs(np.einsum('nij,nji->', dms, m - r)) <= 1e-7
    vj, vk = torch.empty_like(d), torch.empty_like(d)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.lib().jk_build_noalloc(opt.plan, d.data_ptr(), 2, 1, 1, 1, vj.data_ptr(),
                                           vk.data_ptr(), 0.0, st), 'jk_build_noalloc')
    opt.sync()
    same(vj, rj)
    same(vk, rk)
    got = VHFOpt(mol, 1e-16).build().jk_energy_per_atom(d, 1.0, 0.2).cpu().numpy()
    ref, _ = oracle.grad_jk_fast(mol, dms, 1.0, 0.2, tol=0)
    assert np.abs(got - ref).max() <= 1e-10 * np.abs(ref).max()


class _Shifted:
    """A molecule whose AOs start at the third row of its matrices."""

    def __init__(self, mol):
        self._mol = mol

    def __getattr__(self, name):
        return getattr(self._mol, name)

    def ao_loc_nr(self, cart=True):
        return np.asarray(self._mol.ao_loc_nr(cart=cart)) + 3


@pytest.mark.parametrize('hermi', [1, 0])
def test_ao_loc_that_starts_past_zero(torch, hermi):
    """Rows before the first shell belong to no integral: their density is not
    read, their J and K are zero, the rest is as without them."""
    from electrolites_b200.jk import VHFOpt
    mol = clusters.water_mole(2, 4.2, 9, basis='def2-svp')
    n = mol.nao_cart
    d = 0.2 * np.random.default_rng(2).standard_normal((2, n, n))
    if hermi:
        d = d + d.transpose(0, 2, 1)
    big = np.full((2, n + 3, n + 3), 7.0)
    big[:, 3:, 3:] = d
    opt = VHFOpt(_Shifted(mol), TOL).build()
    assert opt.nao == n + 3
    ref = VHFOpt(mol, TOL).build().get_jk(torch.as_tensor(d), hermi)
    for v, r in zip(opt.get_jk(torch.as_tensor(big), hermi), ref):
        assert float((v[:, 3:, 3:] - r).abs().max()) <= ATOL
        assert float(v[:, :3].abs().max()) == 0.0 and float(v[:, :, :3].abs().max()) == 0.0

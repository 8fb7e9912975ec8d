"""The two-role stream kernel where it can go wrong: tiles that hang over every
end of the array, extents below one tile, odd z extents (no aligned rows) and
even ones (16-byte copies with clamped ends), more tiles than CTAs, every
instantiation of the stage (no KO, KO 6, KO 8), all tile shapes (and with them
every shared-memory layout and its barriers) on blocks with and without a ghost
margin, on single blocks and on lists whose CTAs go from block to block; NaN and
infinity, which must stay within the stencil; the calls around the kernel.

Bars as in test_gpu_parity.py: 1e-12 of each field's largest rate (a second
derivative of O(1) data carries eps / h^2 = 2e-14, times at most ~50 terms)."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

H = (0.1, 0.11, 0.09)


def _S(dt=0.02, t=0.7):
    from bssn3d_b200.fused_rhs import pack_S
    return pack_S(2.0, 0.06, dt, H[0], 0.6, 20.0, t, (1, 1, 1, 1), (1, 0), H[1], H[2])


def _state(shape, seed):
    F = 0.05 * np.random.default_rng(seed).standard_normal((24,) + shape)
    for k in (0, 1, 3, 6, 8):
        F[k] += 1.0
    return F


SHAPES = [(1, 1, 1), (2, 3, 5), (4, 4, 16), (5, 3, 17), (3, 9, 18), (8, 4, 33), (23, 26, 34),
          (29, 30, 50), (30, 29, 51)]   # the last two: 256 tiles, more than CTAs


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("ko", [0, 6, 8])
def test_stage_rate_at_tile_edges(shape, ko):
    from bssn3d_b200 import _lib
    lib = _lib.load()
    F, S = _state(shape, sum(shape)), _S()
    sigma = 0.1 if ko else 0.0
    want = O.rhs(F, S) + (O.ko(F, *H, sigma, ko) if ko else 0.0)
    Fd, Sd = torch.from_numpy(F).cuda(), torch.from_numpy(S).cuda()
    acc, nxt = torch.empty_like(Fd), torch.empty_like(Fd)
    _lib.check(lib.bssn_b200_rk4_stage(torch.cuda.current_stream().cuda_stream, 0, Fd.data_ptr(), Fd.data_ptr(),
                                       acc.data_ptr(), nxt.data_ptr(), Sd.data_ptr(), sigma, ko or 6, 1e-4, 1e-4,
                                       *shape))
    got = acc.cpu().numpy()
    assert O.normwise_rel(got, want).max() < 1e-12
    # y_next = u + dt/2 rate, two roundings of O(1) values
    assert np.abs(nxt.cpu().numpy() - (F + 0.5 * S[2] * got)).max() <= 4 * np.finfo(float).eps * np.abs(F).max()


def _one_block(shape, core, variant):
    """A block table of one block (device tensor) and its tile count."""
    import ctypes
    from bssn3d_b200 import _lib
    from bssn3d_b200.amr import BlockDesc
    tab = (BlockDesc * 1)()
    tab[0].sx, tab[0].sy, tab[0].sz = shape
    tab[0].h[:] = H
    tab[0].core = core
    nt = _lib.load().bssn_b200_batch_plan(ctypes.addressof(tab), 1, variant)
    return torch.frombuffer(bytearray(bytes(memoryview(tab).cast("B"))), dtype=torch.uint8).cuda(), nt


# margins below, at and above the stencil's reach; even and odd z extents
@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("core,n", [(0, 13), (1, 18), (1, 13), (2, 16), (2, 17), (3, 10), (3, 17), (4, 12), (5, 11)])
def test_block_tiles_cover_the_core(variant, core, n):
    from bssn3d_b200 import _lib
    lib = _lib.load()
    s = n + 2 * core
    F, S = _state((s, s, s), 7 * n + core), _S()
    S[3] = H[0]                      # a block's dx is its x spacing
    dev, nt = _one_block((s, s, s), core, variant)
    Fd, Sd = torch.from_numpy(F).cuda(), torch.from_numpy(S).cuda()
    out = torch.full_like(Fd, np.nan)
    _lib.check(lib.bssn_b200_batch_rhs(torch.cuda.current_stream().cuda_stream, Fd.data_ptr(), Sd.data_ptr(),
                                       out.data_ptr(), dev.data_ptr(), 1, nt, variant))
    got = out.cpu().numpy()
    inner = (slice(None),) + (slice(core, s - core),) * 3
    written = np.isfinite(got[0])
    assert written.sum() == n ** 3 and written[inner[1:]].all()   # the core and nothing else
    assert O.normwise_rel(got[inner], O.rhs(F, S)[inner]).max() < 1e-12


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("ko,core,n", [(ko, core, n) for ko in (6, 8) for core in (1, 2, 3, 4) for n in (14, 13)]
                         + [(0, 2, 14), (0, 3, 13), (0, 0, 12), (6, 0, 12), (8, 0, 12), (8, 0, 13)])
def test_block_stage_rate_for_every_margin(variant, ko, core, n):
    from bssn3d_b200 import _lib
    lib = _lib.load()
    shape = (n + 2 * core,) * 3
    F, S = _state(shape, 11 * n + core), _S()
    sigma = 0.1 if ko else 0.0
    want = O.rhs(F, S) + (O.ko(F, *H, sigma, ko) if ko else 0.0)
    dev, nt = _one_block(shape, core, variant)
    Fd, Sd = torch.from_numpy(F).cuda(), torch.from_numpy(S).cuda()
    acc, nxt = torch.full_like(Fd, np.nan), torch.full_like(Fd, np.nan)
    _lib.check(lib.bssn_b200_batch_rk4_stage(torch.cuda.current_stream().cuda_stream, 0, Fd.data_ptr(), Fd.data_ptr(),
                                             acc.data_ptr(), nxt.data_ptr(), Sd.data_ptr(), sigma, ko or 6, 1e-4, 1e-4,
                                             dev.data_ptr(), 1, nt, variant))
    got, inner = acc.cpu().numpy(), (slice(None),) + (slice(core, core + n),) * 3
    assert np.isfinite(got).sum() == 24 * n ** 3
    assert O.normwise_rel(got[inner], want[inner]).max() < 1e-12


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("ko", [0, 6, 8])
@pytest.mark.parametrize("margin", [False, True])
def test_block_list_stages_from_block_to_block(variant, ko, margin):
    """Six blocks of unequal shape and spacing, some at odd offsets, in more tiles
    than CTAs: first and last stage against the oracle."""
    import ctypes
    from bssn3d_b200 import _lib
    from bssn3d_b200.amr import BlockDesc
    lib = _lib.load()
    core = 0 if not margin else (4 if ko == 8 else 3)
    inner = [(24, 22, 26), (9, 11, 13), (30, 16, 24), (5, 6, 40), (17, 18, 19), (26, 25, 24)]
    shapes = [tuple(n + 2 * core for n in c) for c in inner]
    tab, at, size = (BlockDesc * len(shapes))(), [], 0
    for b, shape in enumerate(shapes):
        size += b % 2                     # odd offsets for every other pair of blocks
        at.append(size)
        tab[b].offset, tab[b].core = size, core
        tab[b].sx, tab[b].sy, tab[b].sz = shape
        tab[b].h[:] = [h * (1 + 0.25 * b) for h in H]
        size += 24 * int(np.prod(shape))
    nt = lib.bssn_b200_batch_plan(ctypes.addressof(tab), len(shapes), variant)
    assert nt > torch.cuda.get_device_properties(0).multi_processor_count
    dev = torch.frombuffer(bytearray(bytes(memoryview(tab).cast("B"))), dtype=torch.uint8).cuda()
    view = lambda P, b: P[at[b]:at[b] + 24 * int(np.prod(shapes[b]))].reshape((24,) + shapes[b])  # noqa: E731
    Y, U, A = np.zeros(size), np.zeros(size), np.zeros(size)
    for b, shape in enumerate(shapes):
        view(Y, b)[:], view(U, b)[:], view(A, b)[:] = (_state(shape, 31 * b + k) for k in range(3))
    sigma, S = (0.1 if ko else 0.0), _S()
    Sd, Yd, Ud = (torch.from_numpy(x).cuda() for x in (S, Y, U))
    for stage in (0, 3):
        Ad, Od = torch.from_numpy(A).cuda(), torch.full((size,), np.nan, dtype=torch.float64, device="cuda")
        _lib.check(lib.bssn_b200_batch_rk4_stage(
            torch.cuda.current_stream().cuda_stream, stage, Ud.data_ptr(), Yd.data_ptr(), Ad.data_ptr(), Od.data_ptr(),
            Sd.data_ptr(), sigma, ko or 6, 1e-4, 1e-4, dev.data_ptr(), len(shapes), nt, variant))
        acc, out = Ad.cpu().numpy(), Od.cpu().numpy()
        for b, c in enumerate(inner):
            h = [x * (1 + 0.25 * b) for x in H]
            s = S.copy()
            s[3], s[13:16], s[6] = h[0], h, S[6] + (S[2] if stage == 3 else 0.0)
            rate = O.rhs(view(Y, b), s) + (O.ko(view(Y, b), *h, sigma, ko) if ko else 0.0)
            I = (slice(None),) + tuple(slice(core, core + m) for m in c)
            got = view(out, b)
            assert np.isfinite(got).sum() == 24 * np.prod(c)          # the core and nothing else
            if stage == 0:
                assert O.normwise_rel(view(acc, b)[I], rate[I]).max() < 1e-12
                want = view(U, b) + 0.5 * S[2] * rate
            else:
                want = O.enforce(view(U, b) + (S[2] / 6.0) * (view(A, b) + rate))
            assert O.normwise_rel_grouped(got[I], want[I]).max() < 1e-12


@pytest.mark.parametrize("ko", [0, 6, 8])
@pytest.mark.parametrize("shape", [(41, 45, 84), (45, 41, 85)])
def test_derivative_bundle_with_several_tiles_a_cta(shape, ko):
    """792 tiles on 444 CTAs: the hand-over of descriptor and row table, bit for bit."""
    from bssn3d_b200.fused_rhs import derivatives, device_scalars
    F = _state(shape, 5)
    D = derivatives(torch.from_numpy(F).cuda(), device_scalars(_S(), "cuda"), ko_sigma=0.1 if ko else 0.0,
                    ko_order=ko or 6).cpu().numpy()
    np.testing.assert_array_equal(D[:138], O.derivatives(F, *H))
    if ko:
        np.testing.assert_array_equal(D[138:], O.ko(F, *H, 0.1, ko))


@pytest.mark.parametrize("ko", [6, 8])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("field", [1, 4, 2, 9, 13, 22])     # chi, gt, K, beta, At, B: both roles, with and without mixed taps
@pytest.mark.parametrize("shape,at", [((13, 14, 20), (6, 6, 9)), ((13, 14, 21), (12, 13, 20)), ((9, 14, 20), (0, 0, 0)),
                                      ((9, 14, 34), (3, 4, 33))])
def test_nonfinite_values_stay_within_the_stencil(shape, at, field, bad, ko):
    from bssn3d_b200 import _lib
    lib = _lib.load()
    F, Sd = _state(shape, 12), torch.from_numpy(_S()).cuda()
    outs = []
    for value in (F[(field,) + at], bad):
        F[(field,) + at] = value
        Fd = torch.from_numpy(F).cuda()
        acc, nxt = torch.empty_like(Fd), torch.empty_like(Fd)
        _lib.check(lib.bssn_b200_rk4_stage(torch.cuda.current_stream().cuda_stream, 0, Fd.data_ptr(), Fd.data_ptr(),
                                           acc.data_ptr(), nxt.data_ptr(), Sd.data_ptr(), 0.1, ko, 1e-4, 1e-4, *shape))
        outs.append(acc.cpu().numpy())
    # a stencil reaches ko / 2 points along one axis and 3 along two (none of these clamps past the value)
    dist = np.sort(np.abs(np.indices(shape) - np.reshape(at, (3, 1, 1, 1))), axis=0)
    reach = (dist[0] == 0) & (((dist[1] == 0) & (dist[2] <= ko // 2)) | (dist[2] <= 3))
    np.testing.assert_array_equal(outs[1][:, ~reach], outs[0][:, ~reach])
    assert not np.isfinite(outs[1][(field,) + at])


def test_host_scalars_reach_the_device_in_stream_order():
    from bssn3d_b200.fused_rhs import stream_scalars
    want = np.random.default_rng(3).standard_normal(16)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        got = stream_scalars(want, "cuda")
        want_then = want.copy()
        want[:] = 0.0            # read before the call returned
        copy = got.clone()       # ordered after it on the same stream
    side.synchronize()
    assert np.array_equal(copy.cpu().numpy(), want_then)
    with pytest.raises(ValueError):
        stream_scalars(np.zeros(15), "cuda")


@pytest.mark.parametrize("shape,ng", [((9, 9, 9), 3), ((12, 13, 17), 4), ((3, 4, 5), 1), ((40, 11, 66), 3)])
def test_periodic_sync_in_one_pass(shape, ng):
    from bssn3d_b200 import _lib
    F = np.random.default_rng(ng).standard_normal((24,) + shape)
    Fd = torch.from_numpy(F).cuda()
    _lib.check(_lib.load().bssn_b200_periodic_sync(torch.cuda.current_stream().cuda_stream, Fd.data_ptr(), *shape, ng))
    np.testing.assert_array_equal(Fd.cpu().numpy(), O.periodic_sync(F, ng))


def test_rates_take_in_place_operations_with_a_gradient():
    from bssn3d_b200.fused_rhs import cuda_fused_algebra
    from bssn3d_b200.state import FIELD_INPUTS
    shape = (7, 8, 10)
    F = torch.from_numpy(_state(shape, 3)).cuda()
    rates = cuda_fused_algebra({n: F[k] for k, n in enumerate(FIELD_INPUTS)}, *H, 2.0, (1, 1, 1, 1), (1, 0),
                               0.06, 0.02, 0.6, 20.0, 0.7)
    rate = rates["chi"].clone()
    w = torch.full(shape, 2.0, dtype=torch.float64, device="cuda", requires_grad=True)
    rates["chi"].mul_(w)
    rates["chi"].sum().backward()
    assert torch.equal(w.grad, rate)


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
@pytest.mark.parametrize("call", ["rhs_dict", "step", "constraints"])
def test_scalars_are_refused_under_capture(call):
    from bssn3d_b200.constraints import ConstraintSolver
    from bssn3d_b200.evolve import BSSNEvolution
    from bssn3d_b200.grid import Grid
    from bssn3d_b200.rhs import BSSNSolver
    from bssn3d_b200.state import BSSNState
    grid = Grid(Nx=8, Ny=8, Nz=8, dx=0.1, dy=0.1, dz=0.1, ng=3)
    state = BSSNState(torch.from_numpy(_state((14, 14, 14), 2)).cuda())
    fn = {"rhs_dict": lambda: BSSNSolver(grid, dt=0.02, ko_order=6).rhs_dict(state, 0.3, 0.02),
          "step": lambda: BSSNEvolution(grid, ko_sigma=0.1, ko_order=6, bc="none").step(state, 0.3, 0.02).data,
          "constraints": lambda: ConstraintSolver(grid).constraints_tensor(state)}[call]
    fn()
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="captur"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            fn()
    torch.cuda.synchronize()
    fn()


def test_every_enforcement_gives_the_same_bytes():
    from bssn3d_b200 import _lib
    lib = _lib.load()
    shape = (9, 10, 18)
    F, S = _state(shape, 4), _S(dt=1e-300)   # the update itself leaves u as it is
    S[1] = 0.0                                # no CAHD term: it divides by dt
    U, Sd = torch.from_numpy(F).cuda(), torch.from_numpy(S).cuda()
    st = torch.cuda.current_stream().cuda_stream
    n = F[0].size
    want = U.clone()
    _lib.check(lib.bssn_b200_enforce(st, want.data_ptr(), n, 1e-4, 1e-4))
    acc = torch.zeros_like(U)
    fused = torch.empty_like(U)
    _lib.check(lib.bssn_b200_rk4_stage(st, 3, U.data_ptr(), U.data_ptr(), acc.data_ptr(), fused.data_ptr(),
                                       Sd.data_ptr(), 0.0, 6, 1e-4, 1e-4, *shape))
    assert torch.equal(fused, want)
    dev, _ = _one_block(shape, 0, 0)
    D = torch.zeros((138,) + shape, dtype=torch.float64, device="cuda")
    pts = torch.tensor([0, n], dtype=torch.int64, device="cuda")
    out = torch.empty_like(U)
    _lib.check(lib.bssn_b200_batch_rk4_stage_derivs(st, 3, U.data_ptr(), U.data_ptr(), acc.data_ptr(), out.data_ptr(),
                                                    D.data_ptr(), Sd.data_ptr(), 0, 1e-4, 1e-4, dev.data_ptr(), 1,
                                                    pts.data_ptr(), n))
    assert torch.equal(out, want)


def test_enforcement_of_degenerate_metrics():
    """Zero, negative and overflowing determinants come out as the oracle's pow gives them."""
    from bssn3d_b200 import _lib
    F = _state((1, 1, 6), 9)
    F[3:9] = 0.0
    F[3, 0, 0] = [1.0, -1.0, 1e200, -1e200, 0.0, np.nan]
    F[6, 0, 0] = F[8, 0, 0] = [1.0, 1.0, 1e200, 1e200, 0.0, 1.0]
    U = torch.from_numpy(F).cuda()
    _lib.check(_lib.load().bssn_b200_enforce(torch.cuda.current_stream().cuda_stream, U.data_ptr(), 6, 1e-4, 1e-4))
    # 4 ulp: three products and a sum of A~'s trace
    np.testing.assert_allclose(U.cpu().numpy(), O.enforce(F), rtol=4 * np.finfo(float).eps, atol=1e-17)

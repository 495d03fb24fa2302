"""The grouped deposition (particles put into groups, FP64 matrix products)
and the gather by cell against one particle per thread on the same inputs: odd
sizes, each order and pusher, particles in no order and in the guard cells,
exact half-way positions, node changes along every axis, batches that are
not full, crowded cells, and calls that the scratch rules leave alone."""
import numpy as np
import pytest
import torch

from picsar_b200 import _lib
from picsar_b200 import picsar as P

pytestmark = pytest.mark.gpu

G = 4


def _inputs(n, np_, seed, spread):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)
    x = [(r(np_) * (v + 2) - 1) for v in n]                # one cell into the guards
    for a in x:
        a[: np_ // 8] = torch.round(a[: np_ // 8] * 2) / 2  # nodes and half-way points
    u = [spread * (r(np_) - 0.5) for _ in range(3)]
    w = r(np_) + 0.5
    fields = []
    for _ in range(6):
        f = P.grid_zeros(*n, G)
        f.copy_(r(*f.shape) - 0.5)
        fields.append(f)
    return x, u, w, fields


GUARD = 0x5A


def _scratch(query, order, np_, n):
    """The bytes a call asks for, and a pattern behind them."""
    need = _lib.query(query, order, np_, *n, G, G, G)
    assert need > 0
    return torch.full((need + 4096,), GUARD, dtype=torch.uint8, device="cuda"), need


def _thinned(x):
    """Most particles in one octant, so that other groups hold few or none."""
    half = x[0].numel() // 8 * 7
    for a in x:
        a[-half:] = a[-half:] / 2.0
    return x


@pytest.mark.parametrize("order,np_", [(2, 140011), (3, 70001)])
@pytest.mark.parametrize("algo,spread", [(0, 0.4), (1, 1.5)])
def test_deposit_matches_one_particle_per_thread(cuda, order, np_, algo, spread):
    n, dt = (19, 13, 11), 0.5
    x, u, w, _ = _inputs(n, np_, 20 * order + algo, spread)
    x = _thinned(x)
    gi = 1.0 / torch.sqrt(1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    scr, need = _scratch("pxrb_group_scratch", order, np_, n)
    out = []
    for mem in ((None, 0), (scr.data_ptr(), need)):
        j = [P.grid_zeros(*n, G) for _ in range(3)]
        for a in j:
            a.fill_(0.125)                                  # the deposition accumulates
        _lib.call("pxrb_depose_jxjyjz_ws", *[a.data_ptr() for a in j], np_,
                  *[a.data_ptr() for a in x + u], gi.data_ptr(), w.data_ptr(), -1.0, 0.0, 0.0,
                  0.0, dt, 1.0, 1.0, 1.0, *n, G, G, G, order, order, order, algo, err.data_ptr(),
                  *mem, torch.cuda.current_stream().cuda_stream)
        out.append(j)
    assert int(err.item()) == 0
    listed = int(scr[:4].view(torch.int32).item())
    assert 0 < listed < np_                                 # grouped, some on their own
    assert bool((scr[need:] == GUARD).all())
    # a node sums at most the particles of the 5^3 cells around it (8 times the
    # mean in the dense octant): two orders of the sum differ by at most twice
    # that many terms times 2^-53 of the terms' sizes together, for which the
    # largest current is the stricter stand-in (the terms partly cancel)
    terms = 125 * 8 * np_ / (n[0] * n[1] * n[2])
    for a, b in zip(*out):
        assert float((a - b).abs().max()) <= 2 * terms * 2.0 ** -53 * float(b.abs().max())


@pytest.mark.parametrize("order,np_", [(2, 140011), (3, 70001)])
def test_deposit_of_weights_that_are_not_finite(cuda, order, np_):
    """An infinite or NaN weight reaches its particle's own nodes only, as with
    one particle per thread."""
    n = (19, 13, 11)
    x, u, w, _ = _inputs(n, np_, 40 + order, 0.4)
    w[5], w[700], w[1500] = float("inf"), float("nan"), 1e308
    gi = 1.0 / torch.sqrt(1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    scr, need = _scratch("pxrb_group_scratch", order, np_, n)
    out = []
    for mem in ((None, 0), (scr.data_ptr(), need)):
        j = [P.grid_zeros(*n, G) for _ in range(3)]
        _lib.call("pxrb_depose_jxjyjz_ws", *[a.data_ptr() for a in j], np_,
                  *[a.data_ptr() for a in x + u], gi.data_ptr(), w.data_ptr(), -4.0, 0.0, 0.0,
                  0.0, 0.5, 1.0, 1.0, 1.0, *n, G, G, G, order, order, order, 0, err.data_ptr(),
                  *mem, torch.cuda.current_stream().cuda_stream)
        out.append(torch.stack(j))
    a, b = (torch.isfinite(v) for v in out)
    assert not bool(a.all()) and torch.equal(a, b)


@pytest.mark.parametrize("sort", [False, True])
def test_gather_by_cell_is_the_same(cuda, sort):
    """The separate gather with the ordering scratch: the same bits for
    particles in no order, which are taken by cell, and in cell order, which
    are not."""
    n, np_, order = (19, 13, 11), (1 << 20) + 5, 3
    x, u, w, fields = _inputs(n, np_, 30 * order, 0.4)
    if sort:
        by = torch.argsort((torch.floor(x[2]) * 64 + torch.floor(x[1])) * 64 + torch.floor(x[0]))
        x = [a[by].contiguous() for a in x]
    f = [a.data_ptr() for a in fields]
    s = torch.cuda.current_stream().cuda_stream
    scr, need = _scratch("pxrb_order_scratch", order, np_, n)
    out = []
    for mem in ((None, 0), (scr.data_ptr(), need)):
        eb = [torch.full_like(w, 0.25) for _ in range(6)]
        for lower in (0, 1):
            _lib.call("pxrb_geteb3d_energy_conserving_ws", np_, *[a.data_ptr() for a in x],
                      *[a.data_ptr() for a in eb], 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, *n, G, G, G,
                      order, order, order, *f, 0, lower, 64, 0, 0, *mem, s)
        out.append(eb)
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert int(scr[4:8].view(torch.int32).item()) == int(not sort)     # the probe's answer
    assert bool((scr[need:] == GUARD).all())


def _calls(n, np_, order, x, u, w, fields, scr):
    """The deposition and the gather of one call, on scratch `scr` (bytes)."""
    gi = 1.0 / torch.sqrt(1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    j = [P.grid_zeros(*n, G) for _ in range(3)]
    eb = [torch.zeros_like(w) for _ in range(6)]
    s = torch.cuda.current_stream().cuda_stream
    _lib.call("pxrb_depose_jxjyjz_ws", *[a.data_ptr() for a in j], np_,
              *[a.data_ptr() for a in x + u], gi.data_ptr(), w.data_ptr(), -1.0, 0.0, 0.0, 0.0,
              0.5, 1.0, 1.0, 1.0, *n, G, G, G, order, order, order, 0, err.data_ptr(),
              scr.data_ptr(), scr.numel(), s)
    _lib.call("pxrb_geteb3d_energy_conserving_ws", np_, *[a.data_ptr() for a in x],
              *[a.data_ptr() for a in eb], 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, *n, G, G, G, order,
              order, order, *[a.data_ptr() for a in fields], 0, 1, 64, 0, 0, scr.data_ptr(),
              scr.numel(), s)


@pytest.mark.parametrize("order,np_", [(1, 200003), (2, 20011), (3, 20011), (3, 1)])
def test_ample_scratch_does_not_change_the_rule(cuda, order, np_):
    """A call for which the queries ask for no scratch leaves any it is given
    alone, however large."""
    n = (19, 13, 11)
    x, u, w, fields = _inputs(n, np_, 50 + order, 0.4)
    for q in ("pxrb_group_scratch", "pxrb_order_scratch"):
        assert _lib.query(q, order, np_, *n, G, G, G) == 0
    scr = torch.full((1 << 24,), GUARD, dtype=torch.uint8, device="cuda")
    _calls(n, np_, order, x, u, w, fields, scr)
    assert bool((scr == GUARD).all())


def _median_ms(f):
    f()
    took = []
    for _ in range(5):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        took.append(a.elapsed_time(b))
    return sorted(took)[2]


@pytest.mark.parametrize("order,cells", [(2, 1), (2, 10), (3, 1), (3, 10), (3, 1000)])
def test_deposit_of_a_crowded_plasma(cuda, order, cells):
    """2^20 particles in few cells through the public routine: the current of
    one particle per thread, and in no more time (a warp per group took 7 to
    10 times as long in one cell)."""
    n, np_ = (64, 60, 56), 1 << 20
    g = torch.Generator(device="cuda")
    g.manual_seed(cells)
    r = lambda: torch.rand(np_, generator=g, device="cuda", dtype=torch.float64)
    corner = [(torch.rand(cells, generator=g, device="cuda") * (v - 1)).floor() for v in n]
    pick = (r() * cells).long()
    x = [c[pick].double() + r() for c in corner]
    u = [0.2 + 0.05 * r() for _ in range(3)]
    w = r() + 0.5
    gi = 1.0 / torch.sqrt(1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert _lib.query("pxrb_group_scratch", order, np_, *n, G, G, G) > 0
    js = [[P.grid_zeros(*n, G) for _ in range(3)] for _ in range(2)]
    geom = (0.0, 0.0, 0.0, 0.5, 1.0, 1.0, 1.0, *n, G, G, G, order, order, order)

    def grouped():
        P.depose_jxjyjz(*js[0], np_, *x, *u, gi, w, -1.0, *geom, 0, err_flag=err)

    def single():
        _lib.call("pxrb_depose_jxjyjz", *[a.data_ptr() for a in js[1]], np_,
                  *[a.data_ptr() for a in x + u], gi.data_ptr(), w.data_ptr(), -1.0, *geom, 0,
                  err.data_ptr(), torch.cuda.current_stream().cuda_stream)

    grouped()
    single()
    # currents of one sign: two sums of at most np_ terms, each within
    # np_ * 2^-53 of its value
    for a, b in zip(*js):
        assert float((a - b).abs().max()) <= 2 * np_ * 2.0 ** -53 * float(b.abs().max())
    assert int(err.item()) == 0
    assert _median_ms(grouped) <= _median_ms(single)


def _shuffled(n, np_, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda: torch.rand(np_, generator=g, device="cuda", dtype=torch.float64)
    x = [r() * v for v in n]
    u = [0.1 + 0.05 * r() for _ in range(3)]
    w = r() + 0.5
    return x, u, w, 1.0 / torch.sqrt(1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)


@pytest.mark.parametrize("lower", [False, True])
def test_public_gather_of_unsorted_particles(cuda, lower):
    """geteb3d_energy_conserving above its rule's size: the bits of the entry
    that takes no scratch (several scan chunks, grids that stride)."""
    n, np_ = (64, 60, 56), (1 << 20) + 77
    x, u, w, _ = _shuffled(n, np_, 3)
    fields = []
    for q in range(6):
        f = P.grid_zeros(*n, G)
        f.copy_(torch.randn(*f.shape, device="cuda", dtype=torch.float64))
        fields.append(f)
    assert _lib.query("pxrb_order_scratch", 3, np_, *n, G, G, G) > 0
    a, b = ([torch.full_like(w, 0.5) for _ in range(6)] for _ in range(2))
    geom = (0.0, 0.0, 0.0, 1.0, 1.0, 1.0, *n, G, G, G, 3, 3, 3)
    P.geteb3d_energy_conserving(np_, *x, *a, *geom, *fields, False, lower, 64, 0)
    _lib.call("pxrb_geteb3d_energy_conserving", np_, *[v.data_ptr() for v in x + b], *geom,
              *[f.data_ptr() for f in fields], 0, int(lower), 64, 0, 0,
              torch.cuda.current_stream().cuda_stream)
    for p, q in zip(a, b):
        assert torch.equal(p, q)


@pytest.mark.parametrize("order", [2, 3])
def test_public_deposition_with_and_without_memory(cuda, order, monkeypatch):
    """depose_jxjyjz above its rule's size gives one current with scratch and,
    when none can be had, without."""
    n, np_ = (40, 36, 33), 1 << 20
    x, u, w, gi = _shuffled(n, np_, 4)
    assert _lib.query("pxrb_group_scratch", order, np_, *n, G, G, G) > 0
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def deposit():
        j = [P.grid_zeros(*n, G) for _ in range(3)]
        P.depose_jxjyjz(*j, np_, *x, *u, gi, w, -1.0, 0.0, 0.0, 0.0, 0.5, 1.0, 1.0, 1.0, *n, G, G,
                        G, order, order, order, 0, err_flag=err)
        return j

    a, asked = deposit(), []

    def no_memory(*size, **kw):
        asked.append(size)
        raise torch.cuda.OutOfMemoryError("none left")

    monkeypatch.setattr(torch, "empty", no_memory)
    b = deposit()
    assert len(asked) == 1 and int(err.item()) == 0
    # currents of one sign: sums of at most 125 cells' particles
    terms = 125 * np_ / (n[0] * n[1] * n[2])
    for p, q in zip(a, b):
        assert float((p - q).abs().max()) <= 2 * terms * 2.0 ** -53 * float(q.abs().max())

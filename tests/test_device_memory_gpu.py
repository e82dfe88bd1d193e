"""What a case takes of the device's memory: the tables of one-launch stages
only where they are used and where they leave room for other cases."""
import numpy as np
import pytest

import flurrypp_b200 as fb
from flurrypp_b200.decks import write_deck

pytestmark = pytest.mark.gpu

MB = 1 << 20


def box(tmp_path, n, order=3):
    o = dict(nDims=len(n), order=order, meshType=1, dt=0.001)
    for name, m in zip("xyz", n):
        o.update({"n" + name: m, name + "min": 0, name + "max": 1.0})
    return write_deck(str(tmp_path / "m.deck"), **o)


def taken(make):
    """(object, device bytes it took)."""
    import torch

    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = make()
    return s, before - torch.cuda.mem_get_info()[0]


def test_parts_of_a_split_case_take_no_tables(tmp_path):
    d = box(tmp_path, (20, 20, 20))
    for make in (lambda: fb.Solver(d), lambda: fb.Shard(d, 2)):  # the context's own memory
        taken(make)
    one, whole = taken(lambda: fb.Solver(d))
    two, plain = taken(lambda: fb.Solver(d, tile_variant=0))
    sh, parts = taken(lambda: fb.Shard(d, 2))
    assert whole > 1.3 * plain  # the tables, which the parts leave out
    assert parts < 1.1 * plain + 32 * MB


def test_a_second_case_fits_beside_the_first(tmp_path):
    """With memory for two cases and not for both of their tables, both are set
    up, and run as they do with memory to spare (2-D: bit for bit)."""
    import torch

    d = box(tmp_path, (256, 256))
    U = None
    ends = []

    def end(s):
        nonlocal U
        if U is None:
            U = np.array([1.0, 0.3, 0.1, 2.0]) * (1 + np.random.default_rng(7).uniform(-0.01, 0.01, s.shape))
        s.set_state(U)
        s.run(3)
        return s.get_state()

    for v in (-1, 0):  # the kernels of both forms are loaded
        ends.append(end(fb.Solver(d, tile_variant=v)))
    one, plain = taken(lambda: fb.Solver(d, tile_variant=0))
    two, whole = taken(lambda: fb.Solver(d))
    del one, two
    tables = whole - plain
    assert tables > 0.2 * plain
    torch.cuda.empty_cache()
    left = 2 * plain + tables * 6 // 10
    rest = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        both = [fb.Solver(d), fb.Solver(d)]
        ends += [end(s) for s in both]
        del both
    finally:
        del rest
        torch.cuda.empty_cache()
    for e in ends[1:]:
        assert np.array_equal(e, ends[0])


@pytest.mark.parametrize("prec", [fb.FR_PREC_FP64, fb.FR_PREC_MIXED])
def test_server_counts_what_its_cases_hold(tmp_path, prec):
    """A P-multigrid case large enough for one-launch stages: the bytes the
    server counts are those the device gave (to the 2 MB of its pages), and a
    budget below them and above what the case needs without its tables is
    served without them."""
    import time

    import torch

    d = write_deck(str(tmp_path / "p.deck"), nDims=2, order=2, meshType=1, nx=132, ny=130, xmin=0, xmax=1, ymin=0, ymax=1,
                   dtType=2, CFL=0.3, PMG=1, lowOrder=0, smoothSteps=2, uBound=0.35)
    plain, whole = (taken(lambda: fb.Solver(d, precision=prec, tile_variant=v))[1] for v in (0, -1))
    assert whole > 1.15 * plain

    def serve(budget, max_steps, ic=(fb.IC_UNIFORM, ())):
        srv = fb.Server(budget_bytes=budget, max_inflight=2, check_every=10, precision=prec)
        return srv, srv.submit(d, ic=ic, tol=1e-30, max_steps=max_steps)

    srv, rid = serve(8 << 30, 20)  # loads the kernels
    srv.wait(rid, 120)
    srv.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    srv, rid = serve(8 << 30, 10 ** 6)
    t0, counted = time.time(), 0
    while counted == 0 and time.time() - t0 < 60:
        counted = srv.stats()["inflight_bytes"]
    held = before - torch.cuda.mem_get_info()[0]
    srv.cancel(rid)
    srv.close()
    assert counted >= 0.9 * held - 8 * MB, (counted, held)
    srv, rid = serve(counted - 1, 20)
    srv.wait(rid, 120)
    assert srv.poll(rid)["status"] == 2
    srv.close()

"""A wait that gives up inside a kernel is reported by the call that runs into
it, whichever call that is, and only once: a probe kernel runs one bounded wait
out (~1 ms, on a barrier that nothing completes; nothing hangs and the context
stays usable), the next call returns an error, and the one after it works and
gives the values it gave before."""
import numpy as np
import pytest

import tinyscf
from conftest import BAS, DFBAS, xyz

pytestmark = pytest.mark.gpu
CYCLES = 2_000_000


def _engine(name="water"):
    e = tinyscf.TinySCF(BAS, DFBAS, xyz(name), 60)
    e.s.ene_tol = 1e-8
    e.setup()
    return e


def _density(e):
    q, _ = np.linalg.qr(np.random.default_rng(1).normal(size=(e.s.nbasfuncs, e.s.n_occ)))
    return np.ascontiguousarray(q @ q.T), np.ascontiguousarray(q)


@pytest.mark.parametrize("call", ["build_FockMat", "DIIS", "build_DenMat", "sync_host", "reset_scf", "do_SCF", "set_JK"])
def test_every_call_reports_once(call):
    e = _engine()
    D, C = _density(e)
    J, K = np.eye(e.s.nbasfuncs), np.eye(e.s.nbasfuncs)

    def run():
        if call in ("do_SCF", "DIIS"):
            e.reset_scf()
        elif call != "reset_scf":
            e.set_density(D, C)
        if call == "DIIS":
            e.build_FockMat()
        return (lambda: e.set_JK(J, K)) if call == "set_JK" else getattr(e, call)

    def result():
        e.sync_host()
        return np.array([e.energy]), e.mat("J_mat"), e.mat("K_mat"), e.mat("F_mat"), e.mat("D_mat")

    run()()
    before = result()
    f = run()
    e.wait_probe(CYCLES)
    with pytest.raises(tinyscf.TinySCFError):
        f()
    run()()
    for a, b in zip(before, result()):
        assert np.array_equal(a, b)
    e.free()


def test_set_up_calls_report():
    e = tinyscf.TinySCF(BAS, DFBAS, xyz("water"), 60)
    for call in ("compute_Hcore_Ovlp_mat", "compute_sq_Schwarz_scrvals", "prepare_sparsity", "get_initial_guess",
                 "build_DF_tensor"):
        e.wait_probe(CYCLES)
        with pytest.raises(tinyscf.TinySCFError):
            getattr(e, call)()
        getattr(e, call)()
    e.s.ene_tol = 1e-8
    e.do_SCF()
    e.free()


@pytest.mark.parametrize("mixed", [False, True])
def test_batch_reports(mixed):
    es = [_engine(), _engine()]
    if mixed:
        for e in es:
            e.set_k_precision(tinyscf.K_MIXED)
            e.set_density_solver(tinyscf.DENSITY_REFINE)
    b = tinyscf.TinySCFBatch(es)
    b.do_SCF()
    before = [e.energy for e in es]
    for e in es:
        e.reset_scf()
    es[0].wait_probe(CYCLES)
    with pytest.raises(tinyscf.TinySCFError):
        b.do_SCF()
    for e in es:
        e.reset_scf()
    b.do_SCF()
    assert [e.energy for e in es] == before
    b.free()
    for e in es:
        e.free()


def test_another_handle_is_not_blamed_for_a_reported_wait():
    a, b = _engine(), _engine()
    a.wait_probe(CYCLES)
    with pytest.raises(tinyscf.TinySCFError):
        a.build_FockMat()
    b.build_FockMat()
    w, _ = tinyscf.eigh(np.diag([2.0, 1.0]))
    assert np.array_equal(w, [1.0, 2.0])
    b.wait_probe(CYCLES)
    with pytest.raises(tinyscf.TinySCFError):
        tinyscf.eigh(np.diag([2.0, 1.0, 3.0]))
    a.free()
    b.free()

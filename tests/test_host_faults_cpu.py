"""The library's host code over a stand-in for the CUDA runtime
(tests/fake_cuda.cpp): allocations that fail while the task lists are rebuilt.
No kernel runs; every pointer that a launch, copy or graph replay would read is
checked against the live allocations.  Each case runs in a process of its own,
over the objects of the last build."""
import ctypes
import glob
import os
import subprocess
import sys

import numpy as np
import pytest

if __name__ == "__main__":
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules
from hartreefock_b200.build import BUILD

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda"


@pytest.fixture(scope="module")
def fake_library(tmp_path_factory):
    objects = sorted(glob.glob(os.path.join(BUILD, "*.o")))
    if not objects:
        pytest.skip("no objects: python -m hartreefock_b200.build")
    d = tmp_path_factory.mktemp("fake_cuda")
    lib = str(d / "libhfgpu_fake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-fPIC", f"-I{CUDA}/include", "-c",
                    os.path.join(HERE, "fake_cuda.cpp"), "-o", str(d / "fake.o")], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", lib, str(d / "fake.o"), *objects, f"-L{CUDA}/lib64",
                    "-lcublas", "-lcusolver"], check=True)
    yield lib
    os.remove(lib)


def _load(path):
    L = E.library(path)
    L.fake_complaints.restype = L.fake_log.restype = ctypes.c_char_p
    L.fake_live_bytes.restype = L.fake_peak_bytes.restype = ctypes.c_longlong
    return L


def _sound(L):
    text = L.fake_complaints().decode()
    assert not text, text


# --- cases, each in a child process -------------------------------------------------
def rebuild_survives_failed_allocations(L):
    os.environ["HFG_GROUP_MIN_TASKS"] = "0"
    Z, xyz = molecules.water_cluster(2, seed=1)
    P = np.eye(26)
    for graphs in (False, True):
        for n in range(1, 200):
            eng = E.Engine(Z, xyz, "6-31g")
            eng.set_graphs(graphs)
            for _ in range(3):  # the third replays a graph
                eng.fock_rhf(P)
            L.fake_fail_allocation(n)
            try:
                eng.set_prim_target(8)
                failed = False
            except E.HfgError as e:
                failed = True
                assert e.status == 3, e
            L.fake_fail_allocation(0)
            if failed:
                # nothing to build from: an error, not a launch and not a G
                before = L.fake_launches()
                for call in (lambda: eng.fock_rhf(P), lambda: eng.fock_uhf(P, P), eng.eri_packed):
                    with pytest.raises(E.HfgError):
                        call()
                assert L.fake_launches() == before
                eng.set_prim_target(8)  # with memory again, all is well
            for _ in range(3):
                eng.fock_rhf(P)
            eng.fock_uhf(P, P)
            _sound(L)
            live = L.fake_live_bytes()
            eng.close()
            assert L.fake_live_bytes() < live
            if not failed:
                break
        assert not failed and n > 10


def context_gives_everything_back(L):
    os.environ["HFG_GROUP_MIN_TASKS"] = "0"
    Z, xyz = molecules.water_cluster(2, seed=1)
    for n in range(0, 400):
        start = L.fake_live_bytes()
        L.fake_fail_allocation(n)
        try:
            eng = E.Engine(Z, xyz, "6-31g")
        except E.HfgError:
            eng = None
        L.fake_fail_allocation(0)
        if eng:
            eng.close()
        assert L.fake_live_bytes() == start, n
        _sound(L)
        if n and eng:
            break
    assert n > 10


def contexts_on_two_devices(L):
    """Launches, buffers and handles belong to the context's device, whichever
    one is current when it is called."""
    os.environ["HFG_GROUP_MIN_TASKS"] = "0"
    for path in ("0", "1"):
        os.environ["HFG_WARP_PATH"] = path
        for device in (0, 1):
            Z, xyz = molecules.water_cluster(2, seed=1)
            eng = E.Engine(Z, xyz, "6-31g*", device=device)
            n = eng.nbf
            P, C = np.eye(n), np.eye(n)
            calls = [lambda: eng.set_prim_target(8), lambda: eng.fock_rhf(P), lambda: eng.fock_uhf(P, P),
                     eng.eri_packed, lambda: eng.mp2_rhf(C, np.arange(n, dtype=float), 3),
                     lambda: eng.mp2_uhf(C, np.arange(n, dtype=float), 3, C, np.arange(n, dtype=float), 2)]
            for call in calls:
                L.fake_set_device(1 - device)
                call()
                _sound(L)
            small = E.Engine(*molecules.H2O_README, "sto-3g", device=device)
            L.fake_set_device(1 - device)
            small.spin_orbital_eri(np.eye(small.nbf))
            _sound(L)
            small.close()
            eng.close()


def grouped_runs(L):
    """The runs of the grouped tasks are as long as asked for, inside their lists."""
    Z, xyz = molecules.water_cluster(4, seed=1)
    os.environ["HFG_GROUP_MIN_TASKS"] = "0"
    for run, least, most in ((1, 1, 1), (3, 3, 3), (16, 8, 16), (100, 8, 16)):
        os.environ["HFG_GROUP_RUN"] = str(run)
        eng = E.Engine(Z, xyz, "6-31g*")
        for target in (0, 8, 96):
            eng.set_prim_target(target)
            eng.fock_rhf(np.eye(eng.nbf))
            assert least <= L.fake_longest_run() <= most
            assert sum(c["grouped"] for c in eng.class_profile()) == 8
        _sound(L)
        eng.close()
    # small molecules are not grouped of themselves
    del os.environ["HFG_GROUP_MIN_TASKS"]
    eng = E.Engine(Z, xyz, "6-31g*")
    eng.fock_rhf(np.eye(eng.nbf))
    assert L.fake_longest_run() == 0 and not any(c["grouped"] for c in eng.class_profile())


def precision_contexts_hold_no_grouped_lists(L):
    """Contexts in the precision form hold the lists their builds read; the
    first plain build makes the grouped ones, whole or not at all."""
    Z, xyz = molecules.water_cluster(3, seed=1)
    P = np.eye(57)

    def held(min_tasks, **options):
        os.environ["HFG_GROUP_MIN_TASKS"] = min_tasks
        start = L.fake_live_bytes()
        eng = E.Engine(Z, xyz, "6-31g*", **options)
        return eng, L.fake_live_bytes() - start

    for options in ({"incremental": True}, {"mixed_cutoff": 1e-4}, {"density_screening": True}):
        assert held("0", **options)[1] == held("1000000000", **options)[1]
    assert held("0")[1] > held("1000000000")[1]
    for n in range(1, 100):
        eng, _ = held("0", incremental=True)
        eng.set_graphs(True)
        eng.fock_rhf(P)
        eng.set_incremental(False)
        L.fake_fail_allocation(n)
        try:
            eng.fock_rhf(P)
            failed = False
        except E.HfgError:
            failed = True
        L.fake_fail_allocation(0)
        for _ in range(3):
            eng.fock_rhf(P)
        assert sum(c["grouped"] for c in eng.class_profile()) == 8 and L.fake_longest_run() > 0
        _sound(L)
        eng.close()
        if not failed:
            break
    assert n > 10


def plain_builds_hold_no_compaction_lists(L):
    """A plain grouped build allocates its work-queue counters, not a copy of
    the task lists."""
    os.environ["HFG_GROUP_MIN_TASKS"] = "0"
    eng = E.Engine(*molecules.water_cluster(4, seed=1), "6-31g*")
    eng.set_profiling(True)
    tasks = sum(c["tasks"] for c in eng.class_profile())
    for k in ("(21|11)", "(21|20)", "(21|21)", "(22|10)", "(22|11)", "(22|20)", "(22|21)"):
        eng.set_class_path(k, True)  # no scratch
    start = L.fake_live_bytes()
    eng.fock_rhf(np.eye(eng.nbf))
    matrices = 4 * 8 * eng.nbf ** 2  # P, G, J, K
    assert L.fake_live_bytes() - start < matrices + 4096 < matrices + 16 * tasks
    _sound(L)


def autotuners_time_what_they_set(L):
    """The grid autotuner launches the kernels with a grid cap; the task
    autotuner the grouped ones as builds do, from the queue."""
    os.environ["HFG_GROUP_MIN_TASKS"] = "0"
    eng = E.Engine(*molecules.water_cluster(2, seed=1), "6-31g*")
    P = (ctypes.c_double * eng.nbf ** 2)()
    chosen, n = (ctypes.c_int32 * 500)(), ctypes.c_int32()
    L.fake_clear()
    E._check(L.hfg_autotune(eng._h, P, chosen, 500, ctypes.byref(n), None))
    log = L.fake_log().decode()
    assert n.value > 8 and "eri_class_kernel" in log and "eri_group_kernel" not in log
    L.fake_clear()
    E._check(L.hfg_autotune_tasks(eng._h, P, chosen, 500, ctypes.byref(n), None))
    grouped = [line for line in L.fake_log().decode().splitlines() if "eri_group_kernel" in line]
    assert grouped and all(line.endswith(" queue") for line in grouped)
    _sound(L)


def transform_workspaces_are_given_back(L):
    """Workspaces that idle contexts keep: bounded together, given back to an
    allocation that finds no memory, and gone with their context."""
    Z, xyz = molecules.water_cluster(4, seed=1)
    eps = np.arange(76, dtype=float)
    start = L.fake_live_bytes()
    engines = [E.Engine(Z, xyz, "6-31g*") for _ in range(4)]
    for e in engines:
        e.fock_rhf(np.eye(76))
    none = L.fake_live_bytes()
    for e in engines + engines[:2]:  # 450 MB each
        e.mp2_rhf(np.eye(76), eps, 20)
        assert L.fake_live_bytes() - none <= (1 << 30) + (64 << 20)
    kept = L.fake_live_bytes() - none
    assert kept > 256 << 20  # and kept they are
    L.fake_fail_allocation(1)
    other = E.Engine(Z, xyz, "6-31g*")  # finds no memory at first
    assert L.fake_live_bytes() - none < 64 << 20
    for e in engines:
        e.mp2_rhf(np.eye(76), eps, 20)
    for n in (1, 2, 3, 4, 5, 6):  # a transform that fails leaves its context usable
        for e in engines:
            L.fake_fail_allocation(n)
            try:
                e.mp2_rhf(np.eye(76), eps, 20)
            except E.HfgError:
                pass
            L.fake_fail_allocation(0)
            e.mp2_rhf(np.eye(76), eps, 20)
    other.close()
    for e in engines:
        e.close()
    assert L.fake_live_bytes() == start
    _sound(L)


def admission_counts_the_tables_there_are(L):
    """The serving estimate's bytes per primitive pair are those of the engine's
    records, and the estimate covers a context and its first builds."""
    from hartreefock_b200 import serve
    L.fake_prim_pair_bytes.restype = ctypes.c_longlong
    assert serve.PRIM_PAIR_BYTES == L.fake_prim_pair_bytes()
    for mol, basis in ((molecules.water_cluster(2, seed=1), "6-31g*"), (molecules.alkane(3), "6-31+g**"),
                       (molecules.water_cluster(8, seed=1), "6-31g*")):
        start = L.fake_live_bytes()
        eng = E.Engine(*mol, basis)
        for k in ("(21|11)", "(21|20)", "(21|21)", "(22|10)", "(22|11)", "(22|20)", "(22|21)"):
            eng.set_class_path(k, True)
        eng.fock_rhf(np.eye(eng.nbf))
        assert L.fake_live_bytes() - start < serve.footprint_bytes(*mol, basis)
        eng.close()


def far_quartets_need_no_exponential(L):
    """At the limit of the far form the asymptotic Boys function is off by the
    regularised upper incomplete gamma function Q(m + 1/2, T): about half an ulp."""
    from scipy.special import gammaincc
    L.fake_far_T.restype = ctypes.c_double
    for total in range(9):
        T = L.fake_far_T(total)
        assert max(gammaincc(m + 0.5, T) for m in range(total + 1)) < 1.2e-16


CASES = [f.__name__ for f in (rebuild_survives_failed_allocations, context_gives_everything_back,
                              contexts_on_two_devices, grouped_runs,
                              precision_contexts_hold_no_grouped_lists, plain_builds_hold_no_compaction_lists,
                              autotuners_time_what_they_set, transform_workspaces_are_given_back,
                              admission_counts_the_tables_there_are, far_quartets_need_no_exponential)]


@pytest.mark.parametrize("case", CASES)
def test_host_code(fake_library, case):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), fake_library, case], capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


if __name__ == "__main__":
    globals()[sys.argv[2]](_load(sys.argv[1]))

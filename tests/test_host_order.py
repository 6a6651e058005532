"""The host code of the library over a CUDA runtime without a device
(fake_cudart.cpp): what a handle's set-up queues and copies, in which order,
and what its calls do when an allocation or a kernel fails.  Each script runs
in a process of its own with that runtime preloaded."""
import os
import subprocess
import sys
import textwrap

import pytest

from conftest import PKG, REPO

HEAD = """
import ctypes, os, sys
sys.path.insert(0, {pkg!r})
import numpy as np
import bdc_b200 as bdc
fake = ctypes.CDLL(None)
fake.fake_faults.restype = ctypes.c_char_p
fake.fake_fail_malloc.argtypes = [ctypes.c_size_t]
fake.fake_copies.argtypes = [ctypes.c_int, ctypes.c_size_t]
fake.fake_copies.restype = fake.fake_launches.restype = fake.fake_grid.restype = ctypes.c_long
faults = lambda: fake.fake_faults().decode()
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", f"-I{inc}", "-o", so,
                    os.path.join(REPO, "tests", "fake_cudart.cpp")], check=True)

    def run(script, **env):
        e = {k: v for k, v in os.environ.items() if not k.startswith("BDC_")}
        r = subprocess.run([sys.executable, "-c", HEAD.format(pkg=PKG) + textwrap.dedent(script)],
                           env=dict(e, LD_PRELOAD=so, **env), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return run


@pytest.mark.parametrize("n,k", [(12, 11), (14, 12), (20, 10), (21, 13)])
@pytest.mark.parametrize("pinned", [False, True])
def test_set_up_copies_are_ordered(fake, tmp_path, n, k, pinned):
    """No set-up copy may land on a range that the handle's stream has still
    to clear, with every tuning choice measured and with all of them pinned
    (no measurement waits for the stream then)."""
    tune = tmp_path / "tune.txt"
    make = f"""
        E = bdc.Engine({n}, {k}, engine="factored")
        assert faults() == "", faults()
        E.close()
    """
    fake(make, BDC_TUNE_FILE=str(tune))
    if pinned:
        lines = tune.read_text().splitlines()
        assert {ln.split()[2] for ln in lines} >= {"u", "v", "g"}
        fake(make, BDC_TUNE_FILE=str(tune))
        assert tune.read_text().splitlines() == lines  # everything came from the file


def test_passes_refuse_after_a_device_error(fake):
    """An iteration that ends in a device error leaves no usable iterate: the
    passes return that error too, until a distribution is loaded."""
    fake("""
        E = bdc.Engine(20, 10, engine="factored")
        p = np.full(E.R, 0.5 ** 20)
        lnq = np.zeros(bdc.num_q_slots(10))
        passes = [E.log_q, E.log_w, lambda: E.log_w(lnq), E.divergence, lambda: E.divergence(lnq), E.rate,
                  E.mi_forward, E.mi_backward]

        def status(call):
            try:
                call()
                return 0
            except bdc.BDCError as e:
                return e.status

        for call in passes:
            E.set_p(p)
            fake.fake_fault_in(b"k_fac_finalize", 7)
            numeric = status(lambda: E.iterate(1))
            fake.fake_fault_in(b"", 0)
            assert numeric != 0
            assert status(call) == numeric
        E.set_p(p)
        assert [status(c) for c in passes] == [0] * len(passes)
    """)


def test_every_pass_of_a_momentum_step_runs_over_the_grid(fake):
    """A step whose extrapolated point leaves the exponential's range takes all
    of it again: by as many blocks as the step's own pass."""
    fake("""
        E = bdc.Engine(20, 11, engine="factored")
        E.set_p(np.full(E.R, 0.5 ** 20))
        E.accelerate(12, 0.0)
        assert fake.fake_grid(b"k_acc_extrap") > 100
        assert fake.fake_grid(b"k_acc_setz") == fake.fake_grid(b"k_acc_extrap")
    """)


@pytest.mark.parametrize("cpus", [1, 4])
def test_host_vectors_in_pieces_only_into_fresh_pages(fake, cpus):
    """A vector goes in one copy in either direction, but for a large result
    whose pages are not there yet, where several cores can share the faults."""
    if len(os.sched_getaffinity(0)) < cpus:
        pytest.skip("fewer cores here")
    fake(f"""
        import mmap
        os.sched_setaffinity(0, sorted(os.sched_getaffinity(0))[:{cpus}])
        f64p = ctypes.POINTER(ctypes.c_double)
        L = bdc.library()
        for n in (22, 24):
            E = bdc.Engine(n, 3)
            p = np.random.default_rng(n).random(E.R + 1)[1:]
            fake.fake_clear()
            E.set_p(p)
            assert fake.fake_copies(1, 100000) == 1
            maps = [mmap.mmap(-1, 8 * E.R + 4096, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS) for _ in range(2)]
            used, fresh = [np.frombuffer(m, dtype=np.float64)[3:3 + E.R] for m in maps]
            used[:] = 0.0
            many = -(-8 * E.R // 131072) if n == 24 and {cpus} == 4 else 1
            for out, pieces in ((used, 1), (fresh, many), (fresh, 1)):
                fake.fake_clear()
                assert L.bdc_get_p(E._h, out.ctypes.data_as(f64p), E.R) == 0
                assert fake.fake_copies(2, 1000) == pieces
                assert np.array_equal(out, p)
            E.close()
    """)


@pytest.mark.parametrize("line", ["u 3 64", "v 7 64", "u 3 0", "v 7 -3", "u 0 1", "v 99 2", "g 0 0", "g 99 0"])
def test_tuning_choices_outside_the_candidates_are_measured_anew(fake, tmp_path, line):
    """A tune file of another build, or edited by hand, can name a split or a
    tile shape that the set-up has no room or no kernel for."""
    tune = tmp_path / "tune.txt"
    tune.write_text("20 12 u 3 2\n20 12 v 7 2\n20 12 g 3 0\n20 12 oz 0 0\n20 12 " + line + "\n")
    fake("""
        E = bdc.Engine(20, 12, engine="factored")
        E.set_p(np.full(E.R, 0.5 ** 20))
        E.iterate(1)
        E.close()
        assert faults() == "", faults()
    """, BDC_TUNE_FILE=str(tune))


def test_warm_up_runs_when_a_choice_is_measured(fake, tmp_path):
    """The GPU is brought up before any candidate is timed, also with a tune
    file that holds only other keys or some of the choices; with all of them
    pinned there is nothing to warm up for."""
    def transforms(lines):
        tune = tmp_path / "tune.txt"
        tune.write_text("".join(f"20 12 {ln}\n" for ln in lines))
        return int(fake("""
            E = bdc.Engine(20, 12, engine="factored")
            print(fake.fake_launches(b"k_words_q"))
        """, BDC_TUNE_FILE=str(tune)))

    u, v, rest = "u 3 2", "v 7 2", ["g 3 0", "oz 0 0"]
    assert transforms([u, v] + rest) == 0
    assert transforms(["ul 3 8", "qf 1 0"]) == transforms([])
    assert transforms([u, v, rest[0]]) > 0


def test_divergence_needs_no_memory_of_its_own(fake):
    """Where D in dense order cannot be had, the passes that go by it take the
    count path, which needs no buffer beside the handle's."""
    fake("""
        E = bdc.Engine(20, 12, engine="factored")
        E.set_p(np.full(E.R, 0.5 ** 20))
        lnq = np.zeros(bdc.num_q_slots(12))
        fake.fake_fail_malloc(8 << 19)
        for call in (E.divergence, lambda: E.divergence(lnq), E.log_w, E.rate):
            fake.fake_clear()
            call()
            assert fake.fake_launches(b"k_dpass") == 1 and fake.fake_launches(b"k_mma_ba") == 0
        fake.fake_fail_malloc(ctypes.c_size_t(-1).value)
        fake.fake_clear()
        E.rate()
        assert fake.fake_launches(b"k_dpass") == 0 and fake.fake_launches(b"k_mma_ba") == 1
    """)


@pytest.mark.parametrize("first,second,env", [((28, 2), (26, 2), {}), ((18, 14), (20, 11), {"BDC_G_KERNEL": "ozaki"})])
def test_a_later_handle_leaves_the_shared_memory_limits(fake, first, second, env):
    """A kernel's limit belongs to the process: a handle that needs less must
    not take it from one that needs more."""
    fake(f"""
        A = bdc.Engine{first}
        B = bdc.Engine{second}
        for E in (A, B):
            E.set_uniform()
            E.iterate(1)
            E.divergence()
        assert faults() == "", faults()
    """, **env)


@pytest.mark.parametrize("n,k,launches", [(10, 5, 1), (17, 9, 21)])
def test_profile_of_a_direct_handle_times_a_chain(fake, n, k, launches):
    """Twenty iterations of a small problem are one launch of one CTA, or one
    each after a first one for q; the profile times those and counts both
    passes over the folded matrix."""
    fake(f"""
        E = bdc.Engine({n}, {k}, engine="factored")
        E.set_uniform()
        fake.fake_clear()
        d = E.profile(20)
        assert fake.fake_launches(b"8k_direct") == {launches}
        orbits = len(bdc.canonical_reps({k}))
        assert d["work_main"] == 4.0 * E.R * orbits
        assert d["bytes_main"] == E.R * (2.0 * (-(-orbits // 8) * 8) + 40.0)
        assert d["main_kind"] == 3 and d["launches"] == 1 and d["iters"] == 20
        assert d["ms_iter"] == d["ms_main"] == d["ms_d"] == 5.0 / 20
    """)


@pytest.mark.parametrize("n,k,products", [(13, 12, 0), (14, 12, 0), (22, 1, 0), (14, 13, 1), (19, 9, 1)])
def test_divergence_counts_few_pairs(fake, n, k, products):
    """D of a small problem by the count pass, which is the faster one there,
    also on handles with products."""
    fake(f"""
        E = bdc.Engine({n}, {k}, engine="factored")
        E.set_uniform()
        for call in (E.divergence, E.log_w, E.rate):
            fake.fake_clear()
            call()
            assert fake.fake_launches(b"8k_mma_ba") == {products}
            assert fake.fake_launches(b"7k_dpass") == {1 - products}
    """)


@pytest.mark.parametrize("stop,queued", [(1, 1), (2, 3), (3, 3), (5, 7)])
def test_few_iterations_are_queued_past_a_threshold(fake, stop, queued):
    fake(f"""
        E = bdc.Engine(20, 12, engine="factored")
        E.set_uniform()
        fake.fake_clear()
        fake.fake_stop_after({stop})
        st = E.iterate(64, 1e-13)
        assert st["iters"] == {stop} and st["converged"]
        assert fake.fake_launches(b"14k_fac_finalize") == {queued}
    """)


@pytest.mark.parametrize("n,k,count,products,grid", [(14, 7, 4, 0, 9), (17, 9, 64, 0, 2), (18, 9, 2, 0, 74),
                                                     (18, 9, 3, 1, 0), (21, 2, 4, 1, 0), (20, 10, 2, 1, 0)])
def test_forms_in_a_batch(fake, n, k, count, products, grid):
    """Direct instances of a batch take their share of 148 SMs; the larger ones
    go by the products where more than two run together."""
    fake(f"""
        E = [bdc.Engine({n}, {k}, engine="factored") for _ in range({count})]
        for e in E:
            e.set_uniform()
        B = bdc.Batch(E)
        fake.fake_clear()
        B.iterate(4000)  # (the fake device counts an iteration of one handle for all)
        assert (fake.fake_launches(b"8k_mma_ba") >= 8 * {count}) == bool({products})
        if not {products}:
            assert fake.fake_launches(b"8k_mma_ba") == 0 and fake.fake_grid(b"k_direct") == {grid}
        assert faults() == "", faults()
    """)

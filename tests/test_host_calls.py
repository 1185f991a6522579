"""CPU tests of the host code's CUDA calls: the library's objects linked against a CUDA runtime on host
memory (fake_cudart.cu), which runs what a stream was given as late as CUDA allows, makes calls fail on
demand, and reports what the host code did wrong on the way. No GPU, no kernel runs."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from opendust_gb300 import _build, _lib, workloads
from tests._util import case

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    _build.build()
    objs = [os.path.join(_build.OUT_DIR, s.replace(".cu", ".o")) for s in _build.SOURCES]
    if not all(os.path.exists(o) for o in objs):
        _build.build(force=True)
    d = tmp_path_factory.mktemp("fake_cudart")
    obj, lib = str(d / "fake.o"), str(d / "libfake.so")
    # the guard of the device runtime's header: its weak stubs have the names defined here
    subprocess.run([_build._nvcc(), *_build.NVCC_FLAGS, "-D__CUDA_DEVICE_RUNTIME_API_H__",
                    "-diag-suppress", "20096", "-cudart", "none", "-I", _build.CSRC, "-c",
                    os.path.join(HERE, "fake_cudart.cu"), "-o", obj], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", lib, *objs, obj, "-lpthread"], check=True)
    return lib


@pytest.fixture
def fake(fake_path, monkeypatch):
    monkeypatch.setattr(_lib, "_lib", None)
    lib = _lib.load(fake_path)
    lib.fake_log.restype = lib.fake_faults.restype = ctypes.c_char_p
    lib.fake_reset()
    yield lib
    lib.fake_reset()


def faults(lib):
    return lib.fake_faults().decode().splitlines()


def log(lib):
    return lib.fake_log().decode().splitlines()


def member_case(N=1500, n=24, **kw):
    return case(N=N, n=n, builder=workloads.small_plain, trap=np.zeros(15), **kw)[:3]


@pytest.mark.parametrize("plan", [(256, 2, 7, 512), (256, 2, 7, 1024), (256, 4, 7, 4096), (256, 8, 7, 4096)])
def test_batch_member_with_any_each_pair_once_plan(fake, plan):
    # the batch launches each member's work table with the kernel of that member's shape
    with _lib.Batch() as b:
        s = b.add(*member_case())
        b.add(*member_case(N=600))
        b.member(s).set_pair_plan(*plan)
        b.step(2)
    assert any("k_b_pairs_n3" in x for x in log(fake)) and faults(fake) == []


DIRECTED = [(256, 1, 5, 0), (128, 1, 5, 3), (256, 2, 2, 0), (128, 1, 0, 0)]


@pytest.mark.parametrize("plan", DIRECTED)
def test_batch_member_with_a_directed_plan(fake, plan):
    # the batched directed kernel writes one slab of partial sums per source chunk
    with _lib.Batch() as b:
        s = b.add(*member_case(N=5000))
        b.member(s).set_pair_plan(*plan)
        assert b.member(s).pair_plan()["jsplit"] > 1
        b.step(2)
        b.member(s).set_pair_plan(256, 4, 7)
        b.step(1)
        b.member(s).set_pair_plan(*plan)
        b.step(1)
    assert any("9k_b_pairsE" in x for x in log(fake)) and faults(fake) == []


def test_batch_slabs_leave_no_stale_step_graph(fake):
    # a member that has stepped alone from its graph, then in a batch that gives it more slabs
    with _lib.Batch() as b:
        s = b.add(*member_case(N=3000, n=80))
        m = b.member(s)
        m.set_pair_plan(256, 1, 5)
        m.step(40)
        assert "cudaGraphLaunch" in log(fake)
        b.step(1)
        fake.fake_reset()
        m.step(1)
    assert "cudaGraphInstantiate" in log(fake)


def test_batch_launches_follow_a_member_that_changes_its_plan(fake):
    # after the change the member's pairs are launched by the kernel of its new shape, and by no other
    def pair_kernels(plan):
        fake.fake_reset()
        b.member(s).set_pair_plan(*plan)
        b.step(1)
        return {x.split("12k_b_pairs_n3ILi")[1][0] if "12k_b_pairs_n3ILi" in x else "directed"
                for x in log(fake) if "k_b_pairs" in x}

    with _lib.Batch() as b:
        s = b.add(*member_case(N=9000))
        b.step(1)
        for plan, kernel in (((256, 8, 7, 2048), "8"), ((256, 4, 7, 1024), "4"), ((256, 1, 5, 0), "directed"),
                             ((256, 2, 7, 1024), "2")):
            assert pair_kernels(plan) == {kernel}
        fake.fake_reset()
        b.set_plan(s, 8, 2048)
        b.step(1)
        assert any("12k_b_pairs_n3ILi8" in x for x in log(fake)) and faults(fake) == []


def mixed_batch(b):
    # force intervals 2 and 4: steps with and without the pair launch
    return [b.add(*member_case(N=9000, force_every=k)) for k in (2, 4)]


def test_batch_makes_its_graphs_before_it_steps(fake):
    with _lib.Batch() as b:
        slots = mixed_batch(b)
        fake.fake_reset()
        b.step(8)
        calls = log(fake)
        assert calls.count("cudaGraphInstantiate") == 2 and calls.count("cudaGraphLaunch") == 8
        assert "cudaGraphInstantiate" not in calls[calls.index("cudaEventRecord"):]
        # a graph that cannot be made: no step has been launched
        b.remove(slots[0])
        slots[0] = b.add(*member_case(N=9000, force_every=2))
        fake.fake_reset()
        fake.fake_fail(b"cudaGraphInstantiate", 1)
        with pytest.raises(_lib.OpenDustError):
            b.step(8)
        assert "cudaGraphLaunch" not in log(fake)
        assert b.member(slots[1]).step_index == 8 and b.member(slots[0]).step_index == 0


def test_a_failed_call_does_not_fail_the_next(fake):
    # the error of a failed call stays the thread's last error until it is read, and every kernel
    # launch reports that one: it is read where it is reported
    holder, pos, vel = member_case()
    with _lib.Engine(holder) as eng, _lib.Batch() as b:
        eng.set_state(pos, vel)
        fake.fake_fail(b"cudaMemcpyAsync", 0)
        with pytest.raises(_lib.OpenDustError):
            eng.get_state()
        eng.get_state()
        b.add(holder, pos, vel)
        b.step(1)
        fake.fake_fail(b"cudaGraphLaunch", 0)
        with pytest.raises(_lib.OpenDustError):
            b.step(1)
        b.step(1)


def test_batch_launch_that_fails_midway(fake):
    # the members' step indices count what was launched, as the device's do, so that the next call
    # launches the pair kernels on the steps that evaluate (the fourth here, of interval 4)
    with _lib.Batch() as b:
        s = b.add(*member_case(N=9000, force_every=4))
        fake.fake_fail(b"cudaGraphLaunch", 2)
        with pytest.raises(_lib.OpenDustError):
            b.step(6)
        assert b.member(s).step_index == 2 and log(fake)[-1] == "cudaStreamSynchronize"
        pairs = []
        for _ in range(4):
            fake.fake_reset()
            b.step(1)
            pairs.append(any("k_b_pairs" in x for x in log(fake)))
        assert b.member(s).step_index == 6 and pairs == [False, True, False, False]


@pytest.mark.parametrize("bits,status", [(1, 5), (4, 7)])  # a wait that ran out, a crowded cell
def test_batch_forgets_the_error_of_a_member_that_left(fake, bits, status):
    with _lib.Batch() as b:
        first = b.add(*member_case())
        b.add(*member_case(N=700))
        b.step(1)
        fake.fake_member_error(bits)  # of the first member
        for _ in range(2):            # it stays until the member leaves
            with pytest.raises(_lib.OpenDustError) as e:
                b.step(1)
            assert e.value.status == status
        b.remove(first)
        b.step(1)
        fake.fake_reset()
        b.step(1)
        assert log(fake).count("cudaMemcpyAsync") == 1  # the batch's words alone, no member's


@pytest.mark.parametrize("builder", [workloads.small_plain, workloads.field_chain])
def test_force_snapshot_in_place(fake, builder):
    # the caller's positions are read before anything is written to the forces, also where the upload
    # runs late (page-locked memory, or a host whose pageable memory the device reads itself)
    holder, pos, _ = case(N=8000, n=8, builder=builder, trap=np.zeros(15))[:3]
    with _lib.Engine(holder) as eng:
        fake.fake_reset()
        for n in (8000, 1500, 1):  # forces above and below 128 KB
            x = pos[:n].copy()
            _lib.check(fake.od_force_snapshot(eng.h, _lib._dptr(x), n, _lib._dptr(x)), eng.h)
    assert faults(fake) == []


def test_force_snapshot_that_fails_leaves_the_output(fake):
    holder, pos, _ = case(N=1500, n=8, builder=workloads.field_chain, trap=np.zeros(15))[:3]
    force = np.full_like(pos, 7.0)
    with _lib.Engine(holder) as eng:
        fake.fake_poke(b"9k_mc_sort", 10, 4)  # a crowded cell
        assert fake.od_force_snapshot(eng.h, _lib._dptr(pos), 1500, _lib._dptr(force)) == 7
    assert (force == 7.0).all()


@pytest.mark.parametrize("cutoff_lambda", [None, 2.0])
def test_create_keeps_its_upload_sources(fake, cutoff_lambda):
    # what od_create uploads asynchronously lives until the stream has been waited for
    kw = {} if cutoff_lambda is None else dict(cutoff_distance=cutoff_lambda * 1.2e-3)
    holder, pos, vel = member_case(**kw)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        if cutoff_lambda:
            eng.set_pair_plan(256, 4, 3, 1024)
            eng.set_pair_plan(256, 2, 2)
            eng.set_state(pos, vel)
        eng.step(2)
        eng.get_state()
        eng.collect_flags(pos)
    assert faults(fake) == []


def test_plan_without_memory_keeps_the_present_one(fake):
    # a plan that needs more partial-sum slabs than there is memory for: an error, and the present plan
    # with its slabs goes on
    holder, pos, vel = member_case(N=5000)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        eng.set_pair_plan(256, 1, 0, 2)
        eng.step(1)
        fake.fake_fail(b"cudaMalloc", 0)
        with pytest.raises(_lib.OpenDustError) as e:
            eng.set_pair_plan(256, 1, 0, 8)
        assert e.value.status == 3 and eng.pair_plan()["jsplit"] == 2
        eng.step(1)
    assert faults(fake) == []


@pytest.mark.parametrize("N", [300, 2048, 9000])
def test_autotuner_times_every_shape(fake, N):
    # the default (variant 7) among them at every size, without the kernels that a step does not launch
    holder, pos, vel = member_case(N=N)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        fake.fake_reset()
        eng.autotune(use_cache=False)
        calls = log(fake)
    for mt, ms in ((2, 2), (4, 4), (8, 2)):
        assert any(f"10k_pairs_n3ILi{mt}ELi{ms}E" in x for x in calls), mt
    # the sums are taken out of the accumulators once, of the present state with the plan chosen
    assert sum("k_n3_take" in x or "k_acc_take" in x for x in calls) <= 1


@pytest.mark.parametrize("rows,wanted", [(2000, 5), (2520, 5), (30000, 5), (30000, 1)])
def test_series_reads_are_few_contiguous_copies(fake, rows, wanted):
    # up to 256 KB (2520 rows of one grain) one copy, then one per array and 16 MB: no strided ones,
    # which move 8 or 24 bytes at a time
    holder, pos, vel = member_case(N=300, n=rows)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        eng.step(rows)
        fake.fake_reset()
        a = [np.empty((rows, 3)) for _ in range(5)]
        ptr = [_lib._dptr(x) if m < wanted else None for m, x in enumerate(a)]
        _lib.check(fake.od_get_series(eng.h, 0, rows, *ptr), eng.h)
        calls = log(fake)
    assert "cudaMemcpy2DAsync" not in calls
    assert calls.count("cudaMemcpyAsync") == (1 if rows <= 2520 else wanted)


@pytest.mark.parametrize("N,copies", [(2, 1), (1365, 1), (1366, 2)])
def test_small_state_is_one_copy(fake, N, copies):
    holder, pos, vel = member_case(N=N)
    with _lib.Engine(holder) as eng:
        fake.fake_reset()
        eng.set_state(pos, vel)
        # and the error word; more ions also the word of the device's check
        assert log(fake).count("cudaMemcpyAsync") == (2 if copies == 1 else 4)
        fake.fake_reset()
        eng.get_state()
        assert log(fake).count("cudaMemcpyAsync") == copies and faults(fake) == []


@pytest.mark.parametrize("N", [512, 7680, 7681, 15872, 16384, 32768, 33280])
def test_short_fp32_chains_up_to_2_15_ions(fake, N):
    # an FP32 chain of target sums has 64 terms in a whole 4 x 4 group pair, 32 in one of two parts or
    # with sums added after each half
    holder, pos, vel = member_case(N=N)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        eng.step(1)
    names = [x for x in log(fake) if "10k_pairs_n3I" in x]
    kernel = ("ILi4ELi4ELi4ELb0ELb0E" if N <= 7680 else "ILi4ELi4ELi2ELb0ELb0E" if N < 16384 else
              "ILi4ELi4ELi1ELb0ELb1E" if N <= 32768 else "ILi4ELi4ELi1ELb0ELb0E")
    assert names and all(kernel in x for x in names)


@pytest.mark.parametrize("N", [1000, 2000])
@pytest.mark.parametrize("call,fails", [("force_snapshot", b"launch"), ("collect_flags", b"launch"),
                                        ("set_state", b"launch"), ("get_state", b"cudaMemcpyAsync")])
def test_failed_call_leaves_no_copy_behind(fake, call, fails, N):
    # the caller may free its arrays when the call returns, also when it failed after a copy began
    holder, pos, vel = member_case(N=N)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        for after in range(3):
            a, b = pos.copy(), vel.copy()
            fake.fake_reset()
            fake.fake_fail(fails, after)
            args = dict(set_state=(a, b), get_state=()).get(call, (a,))
            try:
                getattr(eng, call)(*args)
            except _lib.OpenDustError:
                assert log(fake)[-1] == "cudaStreamSynchronize"
            a[:] = b[:] = 0.0
            fake.fake_fail(fails, 1000)
            eng.get_state()
            assert faults(fake) == []


@pytest.mark.parametrize("rows", [100, 30000])
def test_failed_series_read_leaves_no_copy_behind(fake, rows):
    holder, pos, vel = member_case(N=300, n=rows)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        eng.step(rows)
        for after in range(1 if rows == 100 else 5):
            fake.fake_reset()
            fake.fake_fail(b"cudaMemcpyAsync", after)
            with pytest.raises(_lib.OpenDustError):
                eng.series(0, rows)
            assert log(fake)[-1] == "cudaStreamSynchronize"


def test_autotuner_that_fails_leaves_clear_accumulators(fake):
    # K3 would take what a failed timing left there as forces
    holder, pos, vel = member_case(N=3000)
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        for after, variant in ((200, 2), (685, 7)):
            fake.fake_reset()
            fake.fake_fail(b"launch", after)
            with pytest.raises(_lib.OpenDustError):
                eng.autotune(use_cache=False)
            assert eng.pair_plan()["variant"] == variant and log(fake)[-1] == "cudaMemsetAsync"

"""libmdg's host side (mdg_api.cu) on a fake CUDA runtime: what a run leaves behind
when one of its calls fails, and the streams that it takes."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    """mdg_api.o as build() made it, linked with the fake runtime and kernels."""
    from mdpy_gb300 import _lib, build as B

    B.build()
    out = tmp_path_factory.mktemp("fake")
    nvcc, objs = [B._nvcc()] + B.ARCH, [os.path.join(B.OBJ, "mdg_api.o")]
    for src in ("fake_cuda.cpp", "fake_kernels.cu"):
        objs.append(str(out / (src + ".o")))
        subprocess.run(nvcc + B.NVCC_FLAGS + ["-c", os.path.join(HERE, "fake", src), "-o", objs[-1]],
                       check=True)
    so = str(out / "libmdg_fake.so")
    subprocess.run(nvcc + ["-shared", "-o", so] + objs + ["-Xlinker", "-Bsymbolic", "-lcudart"],
                   check=True)
    lib = ctypes.CDLL(so)
    for name, argtypes in _lib.SIGNATURES.items():
        if hasattr(lib, name):
            getattr(lib, name).argtypes = argtypes
    lib.mdg_last_error.restype = ctypes.c_char_p
    lib.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_int]
    lib.fake_calls.argtypes = [ctypes.c_char_p]
    lib.fake_device_step.argtypes = [ctypes.c_void_p]
    lib.fake_device_step.restype = ctypes.c_longlong
    lib.fake_stream.restype = ctypes.c_void_p  # flags: 1 = cudaStreamNonBlocking
    lib.fake_begin_capture.argtypes = lib.fake_end_capture_and_run.argtypes = [ctypes.c_void_p]
    return lib


@pytest.fixture
def fake(fake_lib, monkeypatch):
    from mdpy_gb300 import _lib

    monkeypatch.setattr(_lib, "_lib", fake_lib)
    fake_lib.fake_reset()
    return fake_lib


N = 5


def _system():
    from mdpy_gb300 import _lib

    s = _lib.System(N, 40.0)
    s.set_lj(np.ones((N, 4)))
    s.set_masses(np.ones(N))
    s.nonbonded_config(10.0)
    s.integrator_config(_lib.INTEGRATOR_VERLET, 1.0)
    _restore(s)
    return s, _lib.mask(_lib.TERM_LJ)


def _restore(s):
    s.set_positions(np.zeros((N, 3)))
    s.set_velocities(np.zeros((N, 3)))
    s.step = 0


def _whole(fake, s, steps):
    """The state is that of `steps` whole steps, on the device and on the host."""
    assert s.step == steps
    assert fake.fake_device_step(s.handle) == steps
    assert np.all(s.get_velocities() == float(steps))
    assert s.kinetic_energy() == float(steps)  # the fake's: the first velocity


@pytest.mark.parametrize("step_mode", [False, True])
def test_the_mechanics_of_the_fake(fake, step_mode):
    s, mask = _system()
    s.set_graph_mode(1 if step_mode else 0)
    done = 0
    for n in (1, 3, 45, 2, 250, 7):
        s.integrate(n, mask, want_energy=False)
        done += n
        _whole(fake, s, done)
    s.close()


# the calls that a run depends on, failing early or late: a capture refused for want
# of memory, a graph that does not start, a kernel of a step that does not
@pytest.mark.parametrize("nth", [1, 2, 3, 5])
@pytest.mark.parametrize("call", ["cudaGraphInstantiate", "cudaStreamBeginCapture", "cudaGraphLaunch",
                                  "move", "pack", "nonbonded", "bonded", "count_step", "post", "reorder"])
def test_a_failed_run_leaves_no_kick_behind(fake, call, nth):
    """An error ends a run: the finished steps are whole, and the next run starts
    from the positions and velocities that the program then sets, not from what the
    failed one left pending."""
    s, mask = _system()
    fake.fake_fail(call.encode(), nth)
    failed = False
    try:
        for _ in range(6):
            s.integrate(47, mask, want_energy=False)
    except Exception:
        failed = True
    if failed:
        done = s.step
        assert fake.fake_device_step(s.handle) == done
        if call.startswith("cuda"):  # refused between two steps
            _whole(fake, s, done)
            s.get_forces()
    fake.fake_reset()
    # evaluations between the two runs count no step
    s.compute_forces(mask)
    at = fake.fake_device_step(s.handle)
    assert at == s.step
    _restore(s)
    s.integrate(3, mask, want_energy=False)
    _whole(fake, s, 3)
    s.integrate(40, mask, want_energy=True)
    _whole(fake, s, 43)
    s.close()


def test_a_step_cut_short_leaves_no_forces(fake):
    s, mask = _system()
    s.integrate(2, mask, want_energy=False)
    fake.fake_fail(b"nonbonded", 1)
    with pytest.raises(Exception):
        s.integrate(1, mask, want_energy=False)
    with pytest.raises(Exception, match="no force evaluation"):
        s.get_forces()
    s.close()


def _caller_stream(fake, kind):
    if kind == "legacy":
        return 0x1  # cudaStreamLegacy by its handle: cannot be captured
    return fake.fake_stream(1)


@pytest.mark.parametrize("kind", ["own", "legacy"])
@pytest.mark.parametrize("step_mode", [False, True])
@pytest.mark.parametrize("every", [1, 2])
def test_runs_on_a_callers_stream(fake, kind, step_mode, every):
    s, mask = _system()
    s.set_graph_mode(1 if step_mode else 0)
    s.set_mts(every)
    s.set_stream(_caller_stream(fake, kind))
    for _ in range(5):
        s.compute_forces(mask)
    done = 0
    for n in (3, 9, 9, 9, 45, 250):
        s.integrate(n, mask, want_energy=False)
        done += n
        _whole(fake, s, done)
    assert (fake.fake_calls(b"cudaGraphLaunch") == 0) == (kind == "legacy")
    s.close()


@pytest.mark.parametrize("warm", [False, True])  # without and with graphs kept from before
def test_work_under_a_callers_capture(fake, warm):
    """Evaluations and runs on a stream that the caller is capturing become part of
    the caller's graph, whatever the library would do with them otherwise."""
    s, mask = _system()
    stream = fake.fake_stream(1)
    s.set_stream(stream)
    if warm:
        for _ in range(6):
            s.compute_forces(mask)
            s.integrate(9, mask, want_energy=False)
        _restore(s)
    assert fake.fake_begin_capture(stream) == 0
    for _ in range(5):
        s.compute_forces(mask)
        s.integrate(9, mask, want_energy=False)
    s.integrate(61, mask, want_energy=False)
    assert fake.fake_device_step(s.handle) == 0  # nothing ran yet
    assert fake.fake_end_capture_and_run(stream) == 0
    _whole(fake, s, 106)
    s.integrate(50, mask, want_energy=False)
    _whole(fake, s, 156)
    s.close()


def test_reads_allocate_nothing(fake):
    """Not even the first ones: a program may read while another thread captures, or
    once its own pool holds the memory."""
    s, mask = _system()
    s.compute_forces(mask)
    before = fake.fake_calls(b"cudaMalloc"), fake.fake_calls(b"cudaMallocHost")
    s.get_positions(), s.get_velocities(), s.get_forces(), s.get_energies(), s.kinetic_energy()
    s.check_status()
    assert (fake.fake_calls(b"cudaMalloc"), fake.fake_calls(b"cudaMallocHost")) == before
    s.close()


def test_a_launch_shape_can_be_read_and_written_back(fake):
    s, _ = _system()
    default = s.launch_shape
    assert default["split"] == 0  # by the size of each system
    s.set_launch_shape(split=8, pme_block=64)
    assert s.launch_shape["split"] == 8
    s.set_launch_shape(**default)
    assert s.launch_shape == default
    s.set_launch_shape(pme_block=128)
    assert s.launch_shape == dict(default, pme_block=128)
    with pytest.raises(Exception, match="split"):
        s.set_launch_shape(split=3)
    s.close()


@pytest.mark.parametrize("blocking", [True, False])
def test_a_blocking_stream_is_captured_only_for_runs_that_ask_for_it(fake, blocking):
    """While a stream that synchronises with the legacy stream is being captured, another
    thread's work on the legacy stream fails: evaluations and short runs, which come
    often and ask for no graph, leave such a stream alone."""
    s, mask = _system()
    s.set_stream(fake.fake_stream(0 if blocking else 1))
    for _ in range(8):
        s.compute_forces(mask)
        s.integrate(9, mask, want_energy=False)
    _whole(fake, s, 72)
    assert (fake.fake_calls(b"cudaStreamBeginCapture") == 0) == blocking
    s.integrate(250, mask, want_energy=False)
    _whole(fake, s, 322)
    assert fake.fake_calls(b"cudaStreamBeginCapture") > 0
    s.set_graph_mode(1)
    before = fake.fake_calls(b"cudaGraphLaunch")
    s.integrate(5, mask, want_energy=False)
    _whole(fake, s, 327)
    assert fake.fake_calls(b"cudaGraphLaunch") == before + 5
    s.close()

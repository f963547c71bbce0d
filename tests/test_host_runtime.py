"""The library's host side against a stand-in for the CUDA runtime
(fake_cudart.cpp), on a machine without a GPU: what a call has finished with
when it returns, and what it does where the device refuses something."""
import ctypes as C
import importlib.util
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
PKG = ROOT / "spin-glass_b200"


def _module(name, path):
    spec = importlib.util.spec_from_file_location(name, path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """The package bound to the library's objects linked with the stand-in."""
    build = _module("csg_build", PKG / "build.py")
    missing = [u for u in build._units() if not u[0].exists()]
    build.build_lib(force=bool(missing))
    so = tmp_path_factory.mktemp("fake") / "libcsg_fake.so"
    cuda = pathlib.Path(build.NVCC).resolve().parent.parent if "/" in build.NVCC else pathlib.Path("/usr/local/cuda")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", f"-I{cuda / 'include'}", "-Wl,-Bsymbolic",
                    str(ROOT / "tests" / "fake_cudart.cpp"), *[str(o) for o, _ in build._units()], "-o", str(so)],
                   check=True)
    mod = _module("spin_glass_b200_host", PKG / "__init__.py")
    mod.LIB_PATH = so
    L = mod.lib()
    for name, args, res in (("fake_limit", [C.c_size_t], None), ("fake_capacity", [C.c_size_t], None),
                            ("fake_held", [], C.c_size_t), ("fake_host_blocks", [], C.c_size_t),
                            ("fake_wait", [], None), ("fake_max_cluster", [C.c_int], None),
                            ("fake_refuse_launch", [C.c_int], None),
                            ("fake_kept", [], C.c_size_t), ("fake_pending", [C.c_void_p, C.c_size_t], C.c_size_t)):
        f = getattr(L, name)
        f.argtypes, f.restype = args, res
    return mod


@pytest.fixture
def fake(host):
    L = host.lib()
    yield L
    L.fake_limit(C.c_size_t(-1).value)
    L.fake_capacity(C.c_size_t(-1).value)
    L.fake_max_cluster(16)
    L.fake_refuse_launch(-1)


BETAS = np.linspace(2.0, 0.5, 8)


@pytest.mark.parametrize("words", [1, 2, 3])
def test_checkpoint_calls_are_done_with_the_callers_memory(host, fake, words):
    # room for `words` words of the checkpoint at once: 3, 2 and 1 uploads each way
    L, W = 4, 3
    ref = np.zeros((64 * W, L ** 3), np.uint32)
    with host.Engine(L, W, 2, BETAS, seed=1) as e:
        fake.fake_limit(words * 64 * L ** 3 * 4 + 8)
        e.load_checkpoint(ref, 0)
        assert fake.fake_pending(ref.ctypes.data, ref.nbytes) == 0
        host._check(fake.csg_save_checkpoint(e._h, host._p(ref), ref.size))
        assert fake.fake_pending(ref.ctypes.data, ref.nbytes) == 0


@pytest.mark.parametrize("call,launch", [("save", 1), ("load", 1), ("load", 3), ("load", 5)])
def test_checkpoint_calls_that_fail_are_done_with_the_callers_memory(host, fake, call, launch):
    # a launch is refused after copies of other words were queued
    L, W = 4, 3
    ref = np.zeros((64 * W, L ** 3), np.uint32)
    with host.Engine(L, W, 2, BETAS, seed=1) as e:
        fake.fake_limit(64 * L ** 3 * 4 + 8)
        fake.fake_refuse_launch(launch)
        with pytest.raises(host.CsgError):
            if call == "load":
                e.load_checkpoint(ref, 0)
            else:
                host._check(fake.csg_save_checkpoint(e._h, host._p(ref), ref.size))
        assert fake.fake_pending(ref.ctypes.data, ref.nbytes) == 0


def _stream_call(host, fake):
    """One call of the streaming engine on a caller's buffers, waited for; the bytes kept after it."""
    L = 26
    cfg, _keep = host.make_config(L, 1, 2, BETAS, seed=1)
    spins = np.zeros(2 * BETAS.size * L ** 3, np.uint32)
    bonds = np.zeros(3 * L ** 3, np.uint32)
    host.run_device(cfg, spins.ctypes.data, bonds.ctypes.data, None, 0, 2)
    fake.fake_wait()
    return fake.fake_kept()


def test_kept_scratch_is_given_back(host, fake):
    assert _stream_call(host, fake) > 0  # kept for the next call ...
    host.trim_scratch()                  # ... until the caller wants it
    assert fake.fake_kept() == 0
    for make in (lambda: host.Engine(4, 1, 2, BETAS, seed=1), lambda: host.Server(1 << 30, 2, 16),
                 lambda: host.Batch([dict(L=4, n_words=1, n_copies=2, betas=BETAS, seed=1)])):
        owner = make()
        assert _stream_call(host, fake) > 0
        owner.close()
        assert fake.fake_kept() == 0


def test_kept_scratch_does_not_stand_in_an_engines_way(host, fake):
    kept = _stream_call(host, fake)
    fake.fake_capacity(fake.fake_held() + kept + 1000)
    with host.Engine(4, 1, 1, BETAS, seed=1) as e:
        e.init_lattice()


@pytest.mark.parametrize("words", [0, 1, 2])
def test_checkpoint_calls_on_a_full_device(host, fake, words):
    # the device holds the scratch of no word, one or two of three
    L, W = 4, 3
    ref = np.zeros((64 * W, L ** 3), np.uint32)
    with host.Engine(L, W, 2, BETAS, seed=1) as e:
        fake.fake_limit(words * 64 * L ** 3 * 4)
        e.load_checkpoint(ref, 5)
        assert fake.fake_pending(ref.ctypes.data, ref.nbytes) == 0
        host._check(fake.csg_save_checkpoint(e._h, host._p(ref), ref.size))
        assert fake.fake_pending(ref.ctypes.data, ref.nbytes) == 0
        assert e.get_state()[2] == 5
    assert fake.fake_host_blocks() == 0


@pytest.mark.parametrize("most", [4, 8, 16])  # ascending: plans that were placed are kept
def test_requests_whose_tile_cannot_be_placed_take_the_automatic_plan(host, fake, most):
    # two small requests that share the GPU are given one quad per CTA, clusters of 12
    # and 8, whatever clusters the device can place
    fake.fake_max_cluster(most)
    with host.Server(1 << 30, 4, 16) as srv:
        ids = [srv.submit(20, L=16, n_words=1, n_copies=2, betas=np.linspace(2.0, 0.5, 24), seed=1),
               srv.submit(20, L=12, n_words=1, n_copies=2, betas=np.linspace(2.0, 0.5, 16), seed=2)]
        got = set()
        for _ in range(10):
            got |= set(srv.poll()[0])
        assert got == set(ids)
        for i in ids:
            srv.result(i)

"""The library's host side on a fake CUDA runtime (tests/fake_cudart.cpp, no
device): which copies, memsets and launches it gives to which stream, and what
it has waited for when it returns."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    from grapher_b200 import build
    build.build()  # the objects, when they are not up to date
    objs = [os.path.join(build.BUILD, src + ".o") for src in build.SOURCES]
    out = str(tmp_path_factory.mktemp("fake") / "libgvizcuda_fake.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                    "-I/usr/local/cuda/include", "-o", out,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp")] + objs, check=True)
    return out


@pytest.fixture
def fake(fake_path, monkeypatch):
    from grapher_b200 import _native
    monkeypatch.setattr(_native, "LIB_PATH", fake_path)
    monkeypatch.setattr(_native, "_lib", None)
    lib = _native.lib()
    lib.fake_fail_after.argtypes = [ctypes.c_char_p, ctypes.c_int]
    lib.fake_reset()
    return lib


def _graph(n=300):
    from grapher_b200 import graphs
    a, b = graphs.random_connected(n, 0.0, 3)
    return graphs.to_csr(n, a, b)


def _layout(**params):
    from grapher_b200 import ForceLayout, graphs
    row, col = _graph()
    lay = ForceLayout(row, col, model=1)
    lay.set_params(**params)
    lay.begin(0, positions=graphs.randomize_positions(300, 10.0, 1))
    return lay


@pytest.mark.parametrize("params", [dict(), dict(precision=1), dict(barnesHutEnabled=0),
                                    dict(preventOverlap=1, radiusBase=0.5),
                                    dict(precision=1, barnesHutEnabled=0)])
def test_layout_uploads_are_ordered_before_the_work_that_reads_them(fake, tmp_path, params):
    lay = _layout(**params)
    xy = lay.positions()
    lay.step()
    lay.step_host(xy)
    lay.run_host(xy, 3)
    lay.enqueue_steps(2)
    lay.set_fa2_state(np.zeros(600), 1.0, 1.0)
    lay.run(5, 0.0)
    lay.save_checkpoint(tmp_path / "c", "x")
    lay.load_checkpoint(tmp_path / "c", restore_params=True)
    lay.step()
    lay.exact_repulsion(np.arange(200))
    lay.repulsion()
    lay.close()
    assert fake.fake_unordered() == 0


def test_judge_targets_are_ordered_before_the_kernel(fake):
    lay = _layout()
    fake.fake_reset()
    lay.exact_repulsion(np.arange(7))
    assert fake.fake_unordered() == 0
    # an upload that fails is an error, and nothing runs on what was there before
    from grapher_b200._native import GvizCudaError
    fake.fake_reset()
    fake.fake_fail_after(b"cudaMemcpyAsync", 0)
    with pytest.raises(GvizCudaError):
        lay.exact_repulsion(np.arange(9))
    assert fake.fake_launches() == 0
    lay.close()


def test_model_uploads_are_ordered_before_the_work_that_reads_them(fake):
    from grapher_b200.farfield import FarFieldModel
    rng = np.random.default_rng(1)
    X = rng.normal(size=(300, 10)).astype(np.float32)
    T = rng.normal(size=(300, 2)).astype(np.float32)
    W = np.ones(300, np.float32)
    m = FarFieldModel()
    m.gradient(X, T, W)
    m.train(X, T, W, epochs=2, batch=128)
    m.infer(X)
    lay = _layout()
    m.attach(lay)
    lay.set_params(farField=1, farHubTargets=8, farHubTheta=0.5)
    lay.step()
    lay.judge_far_field()
    lay.close()
    m.close()
    assert fake.fake_unordered() == 0


def test_grip_uploads_are_ordered_before_the_work_that_reads_them(fake):
    from grapher_b200.grip import GripRefiner
    row, col = _graph()
    g = GripRefiner(row, col)
    g.set_positions(np.zeros(600))
    g.set_layer(0, np.arange(300), np.arange(301), np.roll(np.arange(300), 1), np.ones(300))
    g.refine_round()
    g.positions()
    g.close()
    assert fake.fake_unordered() == 0


STEPS = [lambda lay, xy: lay.step(), lambda lay, xy: lay.step_host(xy),
         lambda lay, xy: lay.run_host(xy, 3)]


@pytest.mark.parametrize("step", STEPS)
def test_step_without_memory_for_its_result_does_nothing(fake, step):
    from grapher_b200._native import GvizCudaError
    lay = _layout()
    xy = lay.positions()
    fake.fake_reset()
    fake.fake_fail_after(b"cudaMallocHost", 0)
    with pytest.raises(GvizCudaError) as e:
        step(lay, xy)
    assert e.value.code == -1
    assert fake.fake_launches() == 0 and fake.fake_back_to_host() == 0
    fake.fake_reset()
    step(lay, xy)  # the next one is in order
    assert fake.fake_launches() > 0
    lay.close()


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("call", [b"cudaMemcpyAsync", b"cudaMemcpyAsync to host",
                                  b"cudaGraphLaunch"])
@pytest.mark.parametrize("after", range(16))
def test_failed_step_leaves_no_copy_in_flight(fake, step, call, after):
    from grapher_b200._native import GvizCudaError
    lay = _layout()
    xy = lay.positions()
    fake.fake_reset()
    fake.fake_fail_after(call, after)
    try:
        step(lay, xy)
    except GvizCudaError:
        pass
    assert fake.fake_back_to_host() == 0
    fake.fake_reset()
    lay.close()

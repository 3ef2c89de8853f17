import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


@pytest.fixture(scope="session")
def oracle():
    """The CPU oracles (built here from the reference's sources, or prebuilt where they are absent)."""
    from oracle import oracle as O
    need = [os.path.join(O.HERE, "liboracle.so"), os.path.join(O.HERE, "_ref", "libref_f.so")]
    if not all(os.path.exists(p) for p in need):
        O.build()
    if not O.have_reference():
        restate(O)
    return O


def restate(O):
    """Where the reference is absent: the tables, cameras and boxes that tests only feed to the code under
    test, from the restatements that test_host_restatements.py and test_oracle.py pin against the
    reference where it is present (there, without it, those comparisons are skipped)."""
    import ctypes
    import numpy as np
    import little_renderer_b200 as L
    from little_renderer_b200 import workloads as W

    def table(fn, n, dtype):
        out = np.zeros(n, dtype)
        fn(out.ctypes.data_as(ctypes.c_void_p))
        return out

    def camera(fau, vfov, aspect):
        fau = np.asarray(fau, np.float32).reshape(3, 3)
        return W.camera({"from": fau[0], "at": fau[1], "up": fau[2], "vfov": vfov}, aspect)

    def triangle_bounds(quv):
        quv = np.ascontiguousarray(quv, np.float32).reshape(-1, 9)
        q = quv[:, 0:3]
        corners = np.stack([q, q + quv[:, 3:6], q + quv[:, 6:9]])
        out = np.zeros((quv.shape[0], 8), np.float32)
        out[:, 0:3] = corners.min(0) - np.float32(1e-3)
        out[:, 4:7] = corners.max(0) + np.float32(1e-3)
        return out

    O.blue_noise = lambda: table(L.lib().lrc_default_blue_noise, 4096, np.uint16)
    O.bsdf_tables = lambda: table(L.lib().lrc_default_bsdf_tables, 2112, np.float32)
    O.camera, O.triangle_bounds = camera, triangle_bounds


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """A comparison with the reference's own code is skipped where that code is absent."""
    from oracle import oracle as O
    if not O.have_reference() and (item.path.name == "test_host_restatements.py" or "triangle_bounds" in item.name):
        if "oracle" in item.fixturenames:
            pytest.skip("compares with the reference's code, which is absent here")
    outcome = yield
    if outcome.excinfo and issubclass(outcome.excinfo[0], O.ReferenceAbsent):
        outcome.force_exception(pytest.skip.Exception(str(outcome.excinfo[1])))


@pytest.fixture(scope="session")
def ctx():
    import little_renderer_b200 as L
    return L.Context(0)

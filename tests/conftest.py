import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and libscpgpu.so")
    config.addinivalue_line("markers", "slow: long CPU reference runs")


def gpu_available() -> bool:
    try:
        import ctypes
        cudart = None
        for name in ("libcuda.so.1", "libcuda.so"):
            try:
                cudart = ctypes.CDLL(name)
                break
            except OSError:
                continue
        if cudart is None:
            return False
        n = ctypes.c_int(0)
        if cudart.cuInit(0) != 0:
            return False
        return cudart.cuDeviceGetCount(ctypes.byref(n)) == 0 and n.value > 0
    except Exception:
        return False


@pytest.fixture(scope="session")
def gpu():
    if not gpu_available():
        pytest.fail("GPU test selected but no CUDA device is visible")
    from scp_b200 import native
    native.lib()
    return True


# the config-driven host driver and the SFA reader and writer compile the
# reference tree's headers; without that tree neither is built
DRIVER_BIN = os.path.join(ROOT, "scp_b200", "host", "scp_sim_b200")
NEEDS_DRIVER = {"test_driver_restarts_from_its_snapshot": "sfa", "test_driver_reproduces_qcons_record": None}


def pytest_runtest_setup(item):
    """Tests of the host driver skip where it cannot have been built, as the
    ones beside them that take the `reference` fixture do."""
    need = NEEDS_DRIVER.get(getattr(item, "originalname", item.name), False)
    if need is False:
        return
    import oracle
    if not os.path.exists(DRIVER_BIN) or (need == "sfa" and not os.path.exists(oracle.SFA_TOOL)):
        pytest.skip("host driver or SFA tool not built (they compile the reference tree's headers)")


@pytest.fixture(scope="session")
def reference():
    """The reference's own CPU binary (oracle/_ref, built from the reference
    tree by `make -C oracle ref`); tests that run it skip without it."""
    import oracle
    if not oracle.reference_available():
        pytest.skip("reference binary not built (make -C oracle ref needs the reference tree)")
    return True

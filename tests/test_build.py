"""How the libraries are built (pacuda_b200/build.py)."""
from pacuda_b200 import build


def test_device_code_is_not_compressed():
    """A process's first call into a library waits for compressed device code to be unpacked, and nvcc
    compresses any file's past some megabytes unless told not to."""
    assert "--no-compress" in build.FLAGS and "--no-compress" in build.SG_FLAGS

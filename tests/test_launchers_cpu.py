"""Host side of the launchers against a fake CUDA runtime (fake_cudart.cpp), on the CPU: what they ask of the runtime on
each of several devices of one process."""
import ctypes
import os
import shutil
import subprocess

import pytest

from gpt_from_scratch_b200 import build as native_build
from gpt_from_scratch_b200.ops import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
BUF = 1 << 20           # an aligned address that nothing reads


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA toolkit")
    native_build.build()
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = tmp_path_factory.mktemp("fake") / "libgfs_fake.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-Wl,-Bsymbolic", "-I", include,
                    "-I", str(native_build.CSRC),
                    os.path.join(HERE, "fake_cudart.cpp"), *map(str, sorted(native_build.BUILD_DIR.glob("*.o"))),
                    "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out), mode=os.RTLD_LAZY | os.RTLD_LOCAL)
    _lib._declare(lib)
    return lib


def _strides(n):
    return (ctypes.c_longlong * (3 * n))(*[64, 64, 64] * n)


CALLS = {
    **{f"rmsnorm_bwd {rows} x {H}": lambda lib, rows=rows, H=H: lib.gfs_rmsnorm_bwd(BUF, BUF, BUF, BUF, 0, BUF, 0, BUF, rows, H, 0, 0)
       for rows, H in ((4000, 512), (4000, 1024), (4000, 1032), (4000, 2048), (16, 1544), (16, 2048), (4000, 4096))},
    **{f"rmsnorm_bwd_dropout {H}": lambda lib, H=H: lib.gfs_rmsnorm_bwd_dropout(BUF, BUF, BUF, BUF, 0, BUF, BUF, BUF, 4000, H, 0.1, 1, 0)
       for H in (1024, 2048)},
    "embedding_sort_keys": lambda lib: min(lib.gfs_embedding_sort_keys(BUF, BUF, 8, 4096, 0, 1024, 0), 0),
    **{f"flash {D} x {S}": lambda lib, D=D, S=S: lib.gfs_flash_fwd(BUF, BUF, BUF, BUF, 0, BUF, S, 1, 1, D, _strides(4), 0.1, 1, 0, 0)
       for D, S in ((64, 4096), (128, 128), (128, 65536))},
    **{f"flash_bwd {D}": lambda lib, D=D: lib.gfs_flash_bwd(BUF, BUF, BUF, BUF, BUF, BUF, BUF, BUF, BUF, BUF, 512, 1, 1, D, _strides(8),
                                                            0.1, 1, 0, 0, 0, 0) for D in (64, 128)},
    **{f"linear {M} x {N} x {K}": lambda lib, M=M, N=N, K=K: lib.gfs_linear(BUF, BUF, BUF, 0, M, N, K, K, K, N, 0, 0, 0, 0, 0, 0, 0, 1, 60, 0)
       for M, N, K in ((64, 64, 256), (512, 3072, 768), (16384, 768, 768), (16384, 2048, 2048), (8000, 48, 104))},
}


@pytest.mark.parametrize("call", CALLS)
def test_every_device_of_a_process_is_served(fake, call):
    """The limit on dynamic shared memory belongs to a device: the second one must not rest on the first one's, nor a
    return to the first one on either."""
    for dev in (0, 1, 0, 2):
        fake.fake_set_device(dev)
        before = fake.fake_launches()
        assert CALLS[call](fake) == 0, f"device {dev}"
        assert fake.fake_launches() > before
    fake.fake_set_device(0)


@pytest.mark.parametrize("M,N,K", [(64, 64, 256), (512, 3072, 768), (16384, 2048, 2048), (8000, 48, 104)])
def test_late_wait_is_for_one_launch(fake, M, N, K):
    """Tiles, persistent pairs, persistent CTAs: two late-waiting kernels in a row would be three running at once."""
    assert fake.fake_late_waits(M, N, K) == 0b1001       # first of three launches; early_b stays

"""The library's host-only runtime files against a stand-in for the CUDA runtime
(tests/fake_cudart.cpp): which device is waited for before memory is freed, which buffers of a
caller a kernel may take in place, that a kernel's shared-memory limit
never falls, and that memory the pool keeps fails no allocation. No GPU."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "calculixpp_b200", "csrc")
MB = 1 << 20


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    include = next(p for p in (os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),) if os.path.isdir(p))
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-w", "-Wl,-Bsymbolic", "-I", include, "-x", "c++",
                    os.path.join(HERE, "fake_cudart.cpp"), os.path.join(CSRC, "cxg_pool.cu"), os.path.join(CSRC, "cxg_launch.cu"), "-o", out], check=True)
    return out


@pytest.fixture
def fake(built, tmp_path):
    """A copy of the library of its own: its pools and logs start empty."""
    import shutil
    lib = C.CDLL(shutil.copy(built, tmp_path / "libfake.so"))
    lib.fake_log.restype = C.c_char_p
    lib.t_alloc.argtypes = lib.t_malloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
    lib.t_free.argtypes = [C.c_void_p]
    for f in (lib.t_shape, lib.t_launch):
        f.argtypes = [C.c_void_p, C.c_size_t]
    lib.t_kernel_reads.argtypes = [C.c_int, C.c_void_p]
    lib.t_free_all.argtypes = [C.c_int, C.POINTER(C.c_void_p), C.c_int]
    return lib


def calls(lib):
    got = lib.fake_log().decode().split()
    lib.fake_clear()
    return got


def alloc(lib, nbytes, call="t_alloc"):
    p = C.c_void_p()
    rc = getattr(lib, call)(C.byref(p), nbytes)
    return rc, p


@pytest.mark.parametrize("current", [0, 1])
def test_free_waits_for_the_device_of_the_blocks(fake, current):
    fake.cudaSetDevice(1)
    blocks = [alloc(fake, n * MB) for n in (10, 300)]
    assert all(rc == 0 for rc, _ in blocks)
    fake.cudaSetDevice(current)
    calls(fake)
    fake.t_free_all(1, (C.c_void_p * 3)(*[p for _, p in blocks], None), 3)
    back = ["set@0"] if current == 0 else []
    assert calls(fake) == (["set@1"] if back else []) + ["wait@1", "give@1", "free@1"] + back


def test_only_aligned_memory_of_the_device_is_read_in_place(fake):
    fake.cudaSetDevice(1)
    _, p = alloc(fake, MB)
    assert fake.t_kernel_reads(1, p)
    assert not fake.t_kernel_reads(0, p)             # another device's memory
    assert not fake.t_kernel_reads(1, p.value + 4)   # not a place for doubles
    assert not fake.t_kernel_reads(1, None)
    assert not fake.t_kernel_reads(1, C.cast(C.create_string_buffer(64), C.c_void_p))  # host memory


def test_shared_memory_limit_never_falls(fake):
    """Shapes of one kernel known in any order, and on another thread: every launch goes at once."""
    import threading
    kern = 0x1000
    for smem in (60000, 20000, 100000):
        assert fake.t_shape(kern, smem) == 0
    other = threading.Thread(target=fake.t_shape, args=(kern, 8192))
    other.start()
    other.join()
    assert fake.t_shape(kern, 60000) == 0
    assert calls(fake) == ["limit60000@0", "limit100000@0"]
    for smem in (60000, 100000, 8192):
        assert fake.t_launch(kern, smem) == 0
    assert calls(fake) == ["launch@0"] * 3
    fake.cudaSetDevice(1)  # a limit of its own on every device
    assert fake.t_shape(kern, 20000) == 0 and fake.t_launch(kern, 20000) == 0
    assert calls(fake) == ["set@1", "limit20000@1", "launch@1"]


@pytest.mark.parametrize("call", ["t_alloc", "t_malloc"])
def test_memory_the_pool_keeps_fails_no_allocation(fake, call):
    for _, p in [alloc(fake, 200 * MB) for _ in range(2)]:
        fake.t_free(p)  # 400 of the device's 1024 MB idle in the pool
    calls(fake)
    rc, p = alloc(fake, 900 * MB, call)
    assert rc == 0 and calls(fake) == ["malloc@0", "trim@0", "malloc@0"]
    rc, _ = alloc(fake, 200 * MB, call)
    assert rc != 0  # there is no more: an error, not a second trim
    assert [c.split("@")[0] for c in calls(fake)] == (["pool", "trim", "pool"] if call == "t_alloc" else ["malloc", "trim", "malloc"])

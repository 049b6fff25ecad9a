"""The plain product's launcher on several devices of one process: what belongs to a device (the limit of shared memory, how many
CTAs it holds) is set and asked for on each.  The launcher's host code is linked against a runtime without a device
(fake_cudart.c), its kernels are not run."""
import ctypes
import os
import subprocess

import pytest

from gogguf_b200.csrc import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake")
    fake, plain = str(out / "fake.o"), str(out / "plain.so")
    subprocess.run(["gcc", "-O1", "-c", "-fPIC", "-o", fake, os.path.join(HERE, "fake_cudart.c")], check=True)
    src = os.path.join(os.path.dirname(build.__file__), "gemm_plain.cu")
    subprocess.run([build.find_nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-O0", "-std=c++17", "--shared",
                    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-cudart", "none", "-I", os.path.dirname(src), "-o", plain, src,
                    fake, "-Xlinker", "-Bsymbolic"], check=True)
    p = ctypes.CDLL(plain)
    with open(src) as f:
        p.gg_gemm_plain.argtypes = build.parse_signatures(f.read())["gg_gemm_plain"]
    return p


def test_every_tile_on_every_device(lib):
    plain = fake = lib
    count = lambda name: ctypes.c_int.in_dll(fake, name).value                                  # noqa: E731

    def product(M, N, K):
        return plain.gg_gemm_plain(4096, 0, 4096, 0, 4096, 0, 0, M, N, K, K, N, 0, 0)

    sizes = [(M, N, 2048) for M in (1, 2, 4, 8, 16, 33, 65, 200, 2048) for N in (16, 1024, 4096, 16384)]
    early = {}
    for device in (0, 1, 0, 70, 2, 1):                    # (70: beyond the devices an answer is kept for)
        fake.fake_set_device(device)
        for size in sizes:
            assert product(*size) == 0, (device, size)
            want = early.setdefault((device % 2, size), count("fake_last_early"))
            assert count("fake_last_early") == want
    assert count("fake_launches") == 6 * len(sizes)
    # half the multiprocessors hold half the CTAs: somewhere a grid is resident on one kind of device only
    assert any(early[0, s] and not early[1, s] for s in sizes)
    calls = count("fake_attribute_calls")
    for device in (0, 1, 2):
        fake.fake_set_device(device)
        for size in sizes:
            assert product(*size) == 0
    assert count("fake_attribute_calls") == calls          # known by now

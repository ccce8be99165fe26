"""The library on a CUDA runtime without a GPU (fake_cudart.cpp), for tests of its host side."""
import glob
import os
import subprocess

import pytest

from conftest import PKG, ROOT


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    subprocess.run(["make", "-s", "-j8", "-C", PKG], check=True)
    so = str(tmp_path_factory.mktemp("fake") / "libmodlin_fake.so")
    objs = sorted(glob.glob(os.path.join(PKG, "_build", "*.o")))
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include",
                    "-o", so, os.path.join(ROOT, "tests", "fake_cudart.cpp"), *objs, "-lpthread", "-ldl"], check=True)
    return so

"""The whole library over a CUDA runtime without a GPU (host_cuda/fake_cuda.cpp): its host side
runs, kernels do not, and log() says what was asked of the device."""
import ctypes
import importlib.util
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "vx-rs_b200")


def objects():
    """The library's objects (the folder may hold older ones)."""
    text = open(os.path.join(PKG, "Makefile")).read()
    names = [n for kind in ("CU", "CPP") for n in re.search(rf"^{kind}_SRCS := (.*)$", text, re.M)[1].split()]
    return [os.path.join(PKG, "_build", n.rsplit(".", 1)[0] + ".o") for n in names]


class HostGpu:
    def __init__(self, folder):
        lib = os.path.join(folder, "libvx_sgm.so")
        fake = os.path.join(folder, "fake_cuda.o")
        subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-I/usr/local/cuda/include", "-c",
                        os.path.join(HERE, "host_cuda", "fake_cuda.cpp"), "-o", fake], check=True)
        # The library's own calls bind to its own runtime, whatever else the process has loaded.
        # (First in the link: the kernels register with it while the library is loaded.)
        subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined", "-o", lib, fake,
                        *objects(), "-pthread"], check=True)
        shutil.copy(os.path.join(PKG, "vx_sgm.py"), folder)
        spec = importlib.util.spec_from_file_location("vx_sgm_host", os.path.join(folder, "vx_sgm.py"))
        self.vx = importlib.util.module_from_spec(spec)
        shutil.copy(os.path.join(PKG, "libvx_synth.so"), folder)
        import sys
        sys.modules["vx_sgm_host"] = self.vx
        spec.loader.exec_module(self.vx)
        self._lib = ctypes.CDLL(lib)
        self._lib.fake_log.restype = self._lib.fake_kernels.restype = ctypes.c_char_p
        self.ctx = self.vx.Context(0)

    def log(self):
        """Lines since the last call."""
        return self._lib.fake_log().decode().splitlines()

    def launches(self):
        """Names of the kernels launched since the last call, as their templates' arguments have them:
        packed_kernel<8,8,0,0>."""
        out = []
        for line in self.log():
            if line.startswith("launch "):
                name = subprocess.run(["c++filt", line.split()[1]], capture_output=True, text=True, check=True).stdout
                m = re.search(r"(\w+_kernel)(<[^(]*>)?\(", name)
                out.append(m.group(1) + re.sub(r"\((?:bool|int)\)| ", "", m.group(2) or ""))
        return out

    def kernels(self):
        """Every kernel of the library, demangled."""
        return subprocess.run(["c++filt"], input=self._lib.fake_kernels().decode(), capture_output=True, text=True,
                              check=True).stdout.splitlines()

    def fail(self, pitch=0, pool=0):
        self._lib.fake_fail(pitch, pool)


@pytest.fixture(scope="session")
def host_gpu(tmp_path_factory):
    return HostGpu(str(tmp_path_factory.mktemp("host_gpu")))

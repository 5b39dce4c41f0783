"""CPU: host logic of the corrector's entry points (devices, threads, memory)
on a fake CUDA runtime: tests/corrector_host_check.cpp, linked against the
built libtsuner_b200.so, defines the runtime's functions itself."""
import os
import subprocess

import pytest

import tsuner_b200 as T

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda"


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    lib_dir = os.path.dirname(T.LIB_PATH)
    exe = str(tmp_path_factory.mktemp("corr") / "corrector_host_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-rdynamic", "-I" + CUDA + "/include",
                    "-I" + os.path.join(os.path.dirname(HERE), "include"), os.path.join(HERE, "corrector_host_check.cpp"),
                    "-o", exe, "-L" + lib_dir, "-ltsuner_b200", "-Wl,-rpath," + lib_dir, "-Wl,-rpath," + CUDA + "/lib64",
                    "-L" + CUDA + "/lib64", "-lcudart", "-pthread"], check=True)

    def run(scenario):
        r = subprocess.run([exe, scenario], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("scenario", ["two_devices", "threads"])
def test_every_device_is_set_up(check, scenario):
    check(scenario)


def test_a_prediction_takes_the_memory_it_needs(check):
    check("predict_memory")

"""Host-testable pieces of the native code, compiled and run on the CPU."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nguo-3d_b200", "csrc")


def run(tmp_path, body, *flags):
    (tmp_path / "t.cpp").write_text(body)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, *flags, "-o", exe, str(tmp_path / "t.cpp")])
    return subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()


def test_refused_cooperative_launch_falls_back(tmp_path):
    """Error codes that a cooperative launch can return, as a fake would give them: a refusal leaves the
    system to another path, a fault of the context does not."""
    out = run(tmp_path, r"""
#include <cstdio>
#include <initializer_list>
#include "coop.cuh"
int main() {
  for (cudaError_t e : {cudaErrorCooperativeLaunchTooLarge, cudaErrorLaunchOutOfResources, cudaErrorNotSupported,
                        cudaSuccess, cudaErrorInvalidValue, cudaErrorIllegalAddress, cudaErrorMemoryAllocation})
    std::printf("%d ", mg::coop_refused(e) ? 1 : 0);
}
""", "-I", os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"))
    assert out == ["1", "1", "1", "0", "0", "0", "0"]

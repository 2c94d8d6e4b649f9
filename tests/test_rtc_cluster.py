"""Run-time compilation around a generated model: the cluster kernel compiles
with NVRTC for sm_100a, and a program compiles none of the engine's kernels
that a generated model does not use (they made up two thirds of the time that
preparing such a network took)."""
import re

import pytest

import test_rtc_compile as rtc

nvrtc = rtc.nvrtc
HEAD = "#define BG_GENERATED_MODEL 1\n"
MODEL = rtc._MODEL[:rtc._MODEL.index('extern "C"')]


def _compile(src):
    err, prog = nvrtc.nvrtcCreateProgram(src.encode(), b"gen.cu", 0, [], [])
    assert err == nvrtc.nvrtcResult.NVRTC_SUCCESS
    opts = [b"--gpu-architecture=sm_100a", b"-fmad=false", b"-prec-div=true", b"-prec-sqrt=true", b"-ftz=false",
            b"--std=c++17", b"-lineinfo"]
    (res,) = nvrtc.nvrtcCompileProgram(prog, len(opts), opts)
    _, n = nvrtc.nvrtcGetProgramLogSize(prog)
    log = b" " * n
    nvrtc.nvrtcGetProgramLog(prog, log)
    nvrtc.nvrtcDestroyProgram(prog)
    return res == nvrtc.nvrtcResult.NVRTC_SUCCESS, log.decode(errors="replace")


@pytest.mark.parametrize("scalar,npt,multi,pat", [("double", 1, True, 1), ("float", 4, True, 0), ("double", 2, False, 2)])
def test_generated_cluster_compiles(scalar, npt, multi, pat):
    src = HEAD + rtc._embedded_source() + MODEL + """
extern "C" __global__ void __launch_bounds__(bg::kClusterThreads + 32, 1) bg_gen_cluster(const __grid_constant__ bg::ClusterArgs<%s> a) {
    bg::cluster_body<%s, 3, %d, false, %s, %d, bg::GenModel>(a);
}
""" % (scalar, scalar, npt, "true" if multi else "false", pat)
    ok, log = _compile(src)
    assert ok, log[-4000:]


def test_no_other_kernel_is_compiled():
    src = rtc._embedded_source()
    names = re.findall(r"^static __global__ .*?(k_\w+)\(", src, re.M)
    assert len(names) >= 6
    probe = "".join("namespace bg { __device__ void *bg_probe_%s() { return (void *)%s; } }\n" % (n, n) for n in names)
    ok, log = _compile(HEAD + src + MODEL + probe)
    assert not ok
    for n in names:
        assert 'identifier "%s" is undefined' % n in log, n

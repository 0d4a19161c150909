"""The pose loss's launch code (host part of fk_adjoint.cu), compiled with g++ against a fake CUDA runtime."""

import ctypes
import os
import re
import shutil
import subprocess

import pytest
import torch

from betterrobot_b200 import _lib, synthetic as syn, tree as tr

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")

_FAKE = r"""
#include <stdint.h>
#include <stddef.h>
#include "br_b200.h"
#define __host__
#define __device__
typedef int cudaError_t; typedef void* cudaStream_t;
enum { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
static int fail_attribute_call, attribute_calls, launches[4];
template <class K> cudaError_t cudaFuncSetAttribute(K, int, int) {
  return ++attribute_calls == fail_attribute_call ? cudaErrorInvalidValue : cudaSuccess;
}
template <class K> cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, K, int, size_t) { *n = 1; return cudaSuccess; }
static cudaError_t cudaGetLastError() { return cudaSuccess; }
namespace br {
struct DeviceInfo { int device = 0, sms = 148, max_smem_optin = 232448, smem_per_sm = 233472; size_t l2_bytes = 0; };
static const DeviceInfo& device_info() { static DeviceInfo d; return d; }
constexpr int kWarp = 32;
static int round4(int n) { return (n + 3) & ~3; }
static bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
static bool aligned4(const void* p) { return ((uintptr_t)p & 3) == 0; }
static int validate_tree(const br_tree_t* t) { return t ? BR_OK : BR_EINVAL; }
"""

_KERNELS = r"""
template <bool> static void pose_loss_kernel() {}
template <bool> static void pose_loss_lanes_kernel() {}
"""

_TAIL = r"""
extern "C" void fake_reset(int fail) { fail_attribute_call = fail; attribute_calls = 0; for (int& n : launches) n = 0; }
extern "C" int fake_launches(int which) { return launches[which]; }
extern "C" int static_reserve() { return br::kLanesStatic; }
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("launch")
    src = open(os.path.join(REPO, "betterrobot_b200", "csrc", "fk_adjoint.cu")).read()

    def between(a, b):
        return src[src.index(a):src.index(b, src.index(a))]

    layouts = between("struct LossParams", "template <bool kBackward>") + \
        between("struct LaneLayout", "// A visit record")
    code = src[src.index("// When the lane kernel is taken"):]
    which = iter(range(4))  # the lane kernel's launch, the warp kernel's, the scaling's two
    code = re.sub(r"\w+(?:<\w+>)?<<<.*?>>>\(.*?\);", lambda _: f"++launches[{next(which)}];", code)
    cpp, so = str(d / "launch.cpp"), str(d / "launch.so")
    with open(cpp, "w") as f:
        f.write(_FAKE + layouts + _KERNELS + code + _TAIL)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", f"-I{REPO}/include", cpp, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    for name in ("br_pose_loss", "br_pose_loss_backward", "br_pose_loss_value_grad"):
        getattr(lib, name).restype, getattr(lib, name).argtypes = _lib.SIGNATURES[name]
    return lib


def _calls(lib, B):
    dt = tr.DeviceTree(syn.model_from_spec(syn.humanoid_spec()), torch.device("cpu"))
    ids, p = (ctypes.c_int32 * 12)(*range(12)), 64          # (a pointer that nothing reads)
    return {"loss": lambda: lib.br_pose_loss(dt.ptr, p, B, ids, 12, p, p, 0, p, None, None),
            "backward": lambda: lib.br_pose_loss_backward(dt.ptr, p, None, B, ids, 12, p, p, 0, p, p, None),
            "both": lambda: lib.br_pose_loss_value_grad(dt.ptr, p, B, ids, 12, p, p, 0, -1, p, p, None)}


def test_an_error_of_the_lane_kernel_is_returned(host):
    """... and not taken as 'use the other kernel'."""
    for name, call in _calls(host, 50_000).items():
        if name == "both":                                  # (its kernel was configured by "backward")
            continue
        host.fake_reset(1)
        assert call() == 1 and host.fake_launches(0) == host.fake_launches(1) == 0, name
        host.fake_reset(0)
        assert call() == 0 and (host.fake_launches(0), host.fake_launches(1)) == (1, 0), name


def test_small_batches_take_the_warp_kernel(host):
    for name, call in _calls(host, 8_799).items():
        host.fake_reset(0)
        assert call() == 0 and (host.fake_launches(0), host.fake_launches(1)) == (0, 1), name


def test_static_shared_memory_is_reserved(host):
    """The host's fit against the opt-in limit counts all of the kernel's static arrays."""
    src = open(os.path.join(REPO, "betterrobot_b200", "csrc", "fk_adjoint.cu")).read()
    kernel = src[src.index("pose_loss_lanes_kernel(const br_tree_t tree"):src.index("// out[b, :] = unit[b, :]")]
    sizes = {"unsigned long long": 8, "int": 4, "bool": 1}
    total = 0
    for kind, names in re.findall(r"(?<!extern )__shared__ ([a-z ]+?) (\w+(?:\[\w+\])?(?:, \w+(?:\[\w+\])?)*);", kernel):
        for name in names.split(", "):
            total += sizes[kind] * (64 if name.endswith("[BR_MAX_JOINTS]") else 1) + 8   # 8: alignment
    assert 1280 < total <= host.static_reserve()
    assert all(kernel.count(n) > 2 for n in re.findall(r"(\w+)\[BR_MAX_JOINTS\]", kernel))   # each is used

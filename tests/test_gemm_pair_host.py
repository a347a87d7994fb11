"""Where the tcgen05 product's launcher (csrc/gemm_tcgen05.cu) takes pairs of CTAs, on a fake CUDA runtime of two devices: the source is
compiled and linked against functions that write down what they are asked for and refuse a launch whose shared memory was not allowed on the
current device, as the runtime does."""

import ctypes
import os
import subprocess

import pytest

from paged_llm_rs_b200.csrc import build
from paged_llm_rs_b200.errors import KernelError

FAKE = r"""
#include <cuda_runtime_api.h>
#include <cuda.h>
#include <map>
#include <utility>
extern "C" { int fake_device = 0, fake_room = 72, fake_launches = 0, fake_clusters = 0; }
int pllm_pdl_enabled = 0;
static std::map<std::pair<int, const void*>, int> allowed;
static cudaError_t last = cudaSuccess;
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }
extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaGetDevice(int* d) { *d = fake_device; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) { allowed[{fake_device, f}] = v; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = fake_room; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult*) { *f = (void*)encode; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    const auto at = allowed.find({fake_device, f});
    if (c->dynamicSmemBytes > 48 * 1024 && (at == allowed.end() || (size_t)at->second < c->dynamicSmemBytes)) return last = cudaErrorInvalidValue;
    fake_launches++;
    for (unsigned i = 0; i < c->numAttrs; i++) fake_clusters += c->attrs[i].id == cudaLaunchAttributeClusterDimension;
    return cudaSuccess;
}
}
"""


@pytest.fixture(scope="module")
def linked(tmp_path_factory):
    try:
        nvcc = build.find_nvcc()
    except KernelError as e:
        pytest.skip(str(e))
    at = tmp_path_factory.mktemp("pair")
    (at / "fake.cpp").write_text(FAKE)
    inc = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    subprocess.run([nvcc, *build.NVCC_FLAGS, "-c", os.path.join(build.HERE, "gemm_tcgen05.cu"), "-o", str(at / "gemm.o")], check=True)
    subprocess.run(["g++", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-std=c++17", "-I", inc, str(at / "fake.cpp"), str(at / "gemm.o"), "-o", str(at / "gemm.so")], check=True)
    return at / "gemm.so"


def load(linked, tmp_path):
    own = tmp_path / "own.so"          # (a copy, so that what one test's launcher remembers is not another's)
    own.write_bytes(linked.read_bytes())
    lib = ctypes.CDLL(str(own))
    fn = lib.pllm_gemm_tcgen05
    fn.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 4 + [ctypes.c_float] + [ctypes.c_void_p] * 2
    at = lambda name: ctypes.c_int.in_dll(lib, name)

    def product(device, room, glu):
        at("fake_device").value, at("fake_room").value = device, room
        before = at("fake_launches").value, at("fake_clusters").value
        rc = fn(0x1000, 0x2000000, 0x4000000, 2048, 4096, 1024, glu, 0.0, None, None)
        return rc, at("fake_launches").value - before[0], at("fake_clusters").value - before[1]
    return product


@pytest.mark.parametrize("glu", [0, 1])
def test_pairs_are_launched_on_every_device(linked, tmp_path, glu):
    product = load(linked, tmp_path)
    for device in (0, 1, 0, 1):
        assert product(device, 72, glu) == (0, 1, 1)


@pytest.mark.parametrize("glu", [0, 1])
def test_without_room_for_a_pair_the_products_are_the_one_cta_kernels(linked, tmp_path, glu):
    product = load(linked, tmp_path)
    assert product(0, 0, glu) == (0, 1, 0)
    assert product(1, 72, glu) == (0, 1, 1)

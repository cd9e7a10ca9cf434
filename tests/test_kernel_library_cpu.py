"""Which CUDA sources a model has compiled: every entry point belongs to one source, a source's key follows the headers it
includes, and a model names the sources of its parts and no others."""
import ctypes
import re
import subprocess

import pytest
import torch

from llm_serving_engine_b200.csrc import build
from llm_serving_engine_b200.kernels import library


def test_every_declared_entry_point_belongs_to_one_source():
    owners = {}
    for path in build.sources():
        for name in set(build.exported_names(path)):
            assert name not in owners, f"{name} in {path.stem} and {owners[name]}"
            owners[name] = path.stem
    assert set(library._SIGNATURES) <= set(owners)


def test_declared_argument_types_are_those_of_the_sources():
    kinds = {"int": ctypes.c_int, "long long": ctypes.c_longlong, "float": ctypes.c_float, "unsigned": ctypes.c_uint,
             "unsigned int": ctypes.c_uint, "cudaStream_t": ctypes.c_void_p}
    checked = set()
    for path in build.sources():
        for name, arguments in re.findall(r'extern "C" int\s+(lse_\w+)\s*\(([^)]*)\)', path.read_text()):
            if name not in library._SIGNATURES:
                continue
            want = []
            for argument in re.sub(r"//[^\n]*", "", arguments).split(","):
                words = argument.split()
                if not words or words == ["void"]:
                    continue
                want.append(ctypes.c_void_p if "*" in argument else kinds[" ".join(words[:-1])])
            assert library._SIGNATURES[name] == want, name
            checked.add(name)
    assert checked == set(library._SIGNATURES)


def test_a_sources_key_follows_what_it_includes(tmp_path, monkeypatch):
    monkeypatch.setattr(build, "CSRC", tmp_path)
    (tmp_path / "inner.cuh").write_text("int inner;\n")
    (tmp_path / "outer.cuh").write_text('#include "inner.cuh"\n')
    (tmp_path / "a.cu").write_text('#include "outer.cuh"\n')
    (tmp_path / "b.cu").write_text("int b;\n")
    before = [build._key(tmp_path / name, ["-O3"]) for name in ("a.cu", "b.cu")]
    (tmp_path / "inner.cuh").write_text("int other;\n")
    after = [build._key(tmp_path / name, ["-O3"]) for name in ("a.cu", "b.cu")]
    assert after[0] != before[0] and after[1] == before[1]
    assert build._key(tmp_path / "b.cu", ["-O2"]) != after[1]


def test_an_unknown_source_is_an_error():
    with pytest.raises(build.BuildError, match="no CUDA source"):
        build.library_paths(["no_such_source"], verbose=False)


def test_a_model_names_the_sources_of_its_parts_only():
    from llm_serving_engine_b200.cli import RANDOM_MODELS, tiny_config
    from llm_serving_engine_b200.config import load_config
    from llm_serving_engine_b200.models.decoder import kernel_sources

    known = {path.stem for path in build.sources()}
    needed = {}
    for name in RANDOM_MODELS:
        _, _, spec = load_config(tiny_config(name=name))
        for dtype in (torch.float32, torch.bfloat16):
            sources = kernel_sources(spec, dtype)
            assert sources <= known
            assert ("gemm_f32" in sources) == (dtype == torch.float32) and ("gemm_tcgen05" in sources) == (dtype == torch.bfloat16)
            needed[name] = sources
    assert "delta_memory" in needed["kofipel"] and "delta_memory" not in needed["sebudra"]
    assert {"selective_scan", "short_conv", "mlstm", "tanh_norm"} <= needed["tufevik"]
    assert "elementwise" in needed["givelix"] and "residual_streams" in needed["givelix"] and "moe" not in needed["givelix"]


def test_a_model_names_what_its_steps_choose_by_their_rows():
    """The products and the decode step that only some numbers of rows take are loaded with the model, not by the step that first
    takes them: that may be one that is being captured."""
    from llm_serving_engine_b200.config import load_config
    from llm_serving_engine_b200.models.decoder import kernel_sources

    config = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": 528, "hidden_size": 192, "head_dim": 128,
              "intermediate_size": 320, "num_hidden_layers": 2, "num_attention_heads": 2, "num_key_value_heads": 1,
              "max_position_embeddings": 1024, "rope_theta": 10000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": False}
    for head_dim, dtype, want in ((128, torch.bfloat16, {"decode_layers", "gemm_pairs"}), (64, torch.bfloat16, {"gemm_pairs"}), (128, torch.float32, set())):
        _, _, spec = load_config({**config, "head_dim": head_dim})
        assert kernel_sources(spec, dtype) & {"decode_layers", "gemm_pairs"} == want


def test_libraries_share_the_switch_of_dependent_launches():
    """Two libraries in one process have one switch: built here (nvcc needs no GPU), loaded, compared by address."""
    paths = build.library_paths(["elementwise", "tanh_norm"], verbose=False)
    places = {ctypes.addressof(ctypes.c_int.in_dll(ctypes.CDLL(str(path)), "lse_pdl_enabled")) for path in paths.values()}
    assert len(places) == 1


def test_shared_memory_is_allowed_on_every_device_and_never_lowered(tmp_path):
    """The table that kernels of more than 48 KB of shared memory are kept in, compiled here with calls that are counted in
    place of the runtime's: once per device, again for more, not for less, again after an error, and from eight threads at once
    never down."""
    (tmp_path / "trial.cpp").write_text('''
#include <cstddef>
#include <thread>
#include <vector>
#include "smem_allowance.cuh"
static SmemAllowance one, many;
static int calls = 0;
extern "C" int raise_(int device, int bytes, int err) { int before = calls; one.raise(device, bytes, [&](int) { ++calls; return err; }); return calls - before; }
extern "C" int together() {
  int limit = 0, lowered = 0;      // both under the table's lock
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] { for (int i = 0; i < 1000; ++i) many.raise(0, 50000 + (i * 37 + t * 101) % 5000, [&](int most) { lowered += most < limit; limit = most; return 0; }); });
  for (auto& thread : threads) thread.join();
  return lowered;
}
''')
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", f"-I{build.CSRC}", str(tmp_path / "trial.cpp"), "-o",
                    str(tmp_path / "trial.so")], check=True)
    trial = ctypes.CDLL(str(tmp_path / "trial.so"))
    for device, bytes_, err, calls in ((0, 49152, 0, 0), (0, 70000, 0, 1), (0, 70000, 0, 0), (1, 70000, 0, 1), (0, 60000, 0, 0),
                                       (0, 90000, 7, 1), (0, 90000, 0, 1), (1, 90000, 0, 1), (1, 90000, 0, 0), (70, 90000, 0, 1)):
        assert trial.raise_(device, bytes_, err) == calls, (device, bytes_, err)
    assert trial.together() == 0


def test_the_delta_memorys_scan_is_allowed_its_shared_memory_on_every_device(tmp_path):
    """The launcher, compiled here and linked with a runtime that only keeps books: on a second device, and on one of fewer SMs,
    every launch stays within what that device has been asked to allow (48 KB need no asking, static shared memory included, of which
    these kernels have up to 4), and asks for an SM a block where that device has so many."""
    (tmp_path / "books.cpp").write_text('''
#include <cuda_runtime_api.h>
#include <map>
#include <utility>
static int device, launches, refused, largest;
static std::map<std::pair<int, const void*>, int> allowed;
extern "C" {
int use(int which) { device = which; launches = refused = largest = 0; return 0; }
int refusals() { return launches == 2 ? refused : -1; }
int most() { return largest; }
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* out) { *out = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* out, cudaDeviceAttr, int which) { *out = which == 2 ? 20 : 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute, int bytes) { allowed[{device, kernel}] = bytes; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* kernel, void**) {
  const int bytes = (int)config->dynamicSmemBytes;
  const auto found = allowed.find({device, kernel});
  ++launches;
  if (bytes > largest) largest = bytes;
  if (bytes > 44 * 1024 && (found == allowed.end() || bytes > found->second)) { ++refused; return cudaErrorInvalidValue; }
  return cudaSuccess;
}
}
''')
    nvcc = [build._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC"]
    subprocess.run([*nvcc, "-c", str(build.CSRC / "delta_memory_chunks.cu"), "-o", str(tmp_path / "chunks.o")], check=True)
    subprocess.run([*nvcc, "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic", str(tmp_path / "books.cpp"), str(tmp_path / "chunks.o"),
                    "-o", str(tmp_path / "books.so")], check=True)     # its own runtime, also where another is in the process
    books = ctypes.CDLL(str(tmp_path / "books.so"))
    scan = books.lse_delta_chunk_scan
    scan.argtypes = library._SIGNATURES["lse_delta_chunk_scan"]
    for device, lone in ((0, True), (1, True), (0, True), (2, False), (70, True)):
        for dim in (24, 64, 128, 200):
            books.use(device)
            # q .. beta, z, partials of z, bias and decay, state, segments, results, buffer; 10 chunks of one request, four heads
            assert scan(*[None] * 5, 1, 0, 0, *[None] * 7, 10, 1, 4, 4, dim, 128, 1, 1, None) == 0
            assert books.refusals() == 0, (device, dim)
            assert lone == (books.most() >= 116 * 1024) or dim > 128

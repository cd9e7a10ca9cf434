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


_BOOKS = '''
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <map>
#include <string>
#include <utility>
// A runtime that keeps books and runs nothing.  Device 2 has 20 SMs, device 3 takes no cooperative launches.
static int device, launches, refused, largest, refuse_cooperative, a_sm = 1;
static cudaError_t last = cudaSuccess;
static std::map<std::pair<int, const void*>, int> allowed;
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                       const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
extern "C" {
int use(int which, int blocks_a_sm, int refuse) {
  device = which; launches = refused = largest = 0; a_sm = blocks_a_sm; refuse_cooperative = refuse; last = cudaSuccess;
  return 0;
}
int launched() { return launches; }
int refusals() { return refused; }
int most() { return largest; }
int pending() { return (int)last; }
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* out) { *out = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t was = last; last = cudaSuccess; return was; }
cudaError_t cudaDeviceGetAttribute(int* out, cudaDeviceAttr what, int which) {
  *out = what == cudaDevAttrCooperativeLaunch ? which != 3 : which == 2 ? 20 : 148;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute, int bytes) { allowed[{device, kernel}] = bytes; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* out, const void*, int, size_t, unsigned) { *out = a_sm; return cudaSuccess; }
#undef cudaGetDriverEntryPoint
cudaError_t cudaGetDriverEntryPoint(const char* name, void** out, unsigned long long, cudaDriverEntryPointQueryResult* found) {
  *out = std::string(name) == "cuTensorMapEncodeTiled" ? (void*)encode : nullptr;
  *found = *out ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaErrorUnknown; }
cudaError_t cudaMemcpyFromSymbolAsync(void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaErrorUnknown; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return last = cudaErrorUnknown; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* kernel, void**) {
  const int bytes = (int)config->dynamicSmemBytes;
  const auto found = allowed.find({device, kernel});
  ++launches;
  if (bytes > largest) largest = bytes;
  if (bytes > 44 * 1024 && (found == allowed.end() || bytes > found->second)) { ++refused; return last = cudaErrorInvalidValue; }
  if (config->attrs[0].id == cudaLaunchAttributeCooperative && refuse_cooperative) return last = cudaErrorCooperativeLaunchTooLarge;
  return cudaSuccess;
}
}
'''


def _with_books(source, folder):
    """A source's launchers, compiled here and linked with a runtime that only keeps books."""
    (folder / "books.cpp").write_text(_BOOKS)
    nvcc = [build._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC"]
    subprocess.run([*nvcc, "-c", str(build.CSRC / f"{source}.cu"), "-o", str(folder / "source.o")], check=True)
    subprocess.run([*nvcc, "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic", str(folder / "books.cpp"), str(folder / "source.o"),
                    "-o", str(folder / "books.so")], check=True)     # its own runtime, also where another is in the process
    books = ctypes.CDLL(str(folder / "books.so"))
    for name, types in library._SIGNATURES.items():
        if name in build.exported_names(build.CSRC / f"{source}.cu"):
            getattr(books, name).argtypes = types
    return books


def test_the_delta_memorys_scan_is_allowed_its_shared_memory_on_every_device(tmp_path):
    """On a second device, and on one of fewer SMs, every launch stays within what that device has been asked to allow (48 KB need no
    asking, static shared memory included, of which these kernels have up to 4), and asks for an SM a block where that device has
    so many."""
    books = _with_books("delta_memory_chunks", tmp_path)
    for device, lone in ((0, True), (1, True), (0, True), (2, False), (70, True)):
        for dim in (24, 64, 128, 200):
            books.use(device, 1, 0)
            # q .. beta, z, partials of z, bias and decay, state, segments, results, buffer; 10 chunks of one request, four heads
            assert books.lse_delta_chunk_scan(*[None] * 5, 1, 0, 0, *[None] * 7, 10, 1, 4, 4, dim, 128, 1, 1, None) == 0
            assert books.launched() == 2 and books.refusals() == 0, (device, dim)
            assert lone == (books.most() >= 116 * 1024) or dim > 128


def test_a_device_that_does_not_take_the_one_launch_step_is_asked_and_leaves_no_error(tmp_path):
    """A device without cooperative launches, or one on which not all blocks fit at once, is known when a model is built; a launch
    that is refused all the same (a process that may use a part of the SMs only) says so, and the next launch does not meet its error."""
    books = _with_books("decode_layers", tmp_path)
    sizes = (2, 1, 192, 320, 2, 1, 528)           # layers, rows, hidden, feed-forward, query and key/value heads, vocabulary
    for device, blocks_a_sm, blocks, want in ((0, 1, 148, 1), (0, 0, 148, 0), (3, 1, 148, 0), (2, 1, 148, 0), (2, 1, 20, 1), (0, 1, 20, 1)):
        books.use(device, blocks_a_sm, 0)
        assert books.lse_decode_layers_fits(blocks, *sizes) == want, (device, blocks_a_sm, blocks)
        assert books.pending() == 0
    layers = (ctypes.c_longlong * 18)()
    eps = (ctypes.c_float * 4)()

    def step():
        return books.lse_decode_layers(layers, eps, 2, None, 528, 1.0, None, None, 1e-6, None, 0, None, None, None, None, None, 4, 1, 1, 192,
                                       320, 2, 1, 528, 16, 8, 1.0, None, None, 148, None)
    books.use(0, 1, 0)
    assert step() == 0 and books.launched() == 2 and books.refusals() == 0
    books.use(0, 1, 1)
    assert step() == -3 and books.launched() == 2 and books.pending() == 0

"""The C++ shim's workspaces under several host threads, without a GPU: the shim is compiled against stand-ins for the
reference's Tensor, for the CUDA runtime and for the C ABI, which record whether two calls were ever inside one workspace."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "modern-llm-v1_b200", "csrc")

TENSOR = r"""
#pragma once
#include <cstdint>
#include <cstdlib>
#include <vector>
namespace modernllm {
enum class DType { FP32, BF16 };
enum class Device { Cpu, Cuda };
class Tensor {
public:
    Tensor(std::vector<std::int64_t> shape, DType t, Device d) : n_(1), t_(t), d_(d) {
        for (auto s : shape) n_ *= s;
        mem_.resize(bytes());
    }
    DType dtype() const { return t_; }
    Device device() const { return d_; }
    std::int64_t numel() const { return n_; }
    size_t bytes() const { return size_t(n_) * (t_ == DType::FP32 ? 4 : 2); }
    void* data() { return mem_.data(); }
    const void* data() const { return mem_.data(); }
    template <typename T> T* data_as() { return reinterpret_cast<T*>(mem_.data()); }
    template <typename T> const T* data_as() const { return reinterpret_cast<const T*>(mem_.data()); }
private:
    std::int64_t n_;
    DType t_;
    Device d_;
    std::vector<unsigned char> mem_;
};
}  // namespace modernllm
"""

HARNESS = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <thread>
#include "modernllm_shim.h"
#include "b200attn.h"
using namespace modernllm;
static std::atomic<int> overlaps{0}, calls{0}, in_static{0};
// a call that keeps writing to its workspace for a while: two of them in one workspace see each other
static int use(void* ws, size_t bytes) {
    static std::atomic<unsigned char> next{1};
    const unsigned char mine = next++;
    ++calls;
    for (int i = 0; i < 20; ++i) {
        std::memset(ws, mine, bytes);
        std::this_thread::sleep_for(std::chrono::microseconds(50));
        for (size_t k = 0; k < bytes; ++k)
            if (static_cast<volatile unsigned char*>(ws)[k] != mine) { ++overlaps; return 0; }
    }
    return 0;
}
extern "C" {
int cudaGetDevice(int* d) { *d = 0; return 0; }
int b200attn_fwd(const void*, const void*, const void*, void*, float*, int, int, int, int, int, int, float, void*) { return 0; }
int b200attn_fwd_kvcache(const void*, const void*, const void*, void*, float*, int, int, int, int, int, int, int, float, void*) { return 0; }
int b200attn_bwd_static(const void*, const void*, const void*, const void*, const float*, const void*, void*, void*, void*, int, int, int, int, int, int, float, void*) {
    ++calls;
    if (in_static++ != 0) ++overlaps;
    std::this_thread::sleep_for(std::chrono::milliseconds(1));
    --in_static;
    return 0;
}
size_t b200attn_bwd_workspace_bytes_mode(int B, int T, int Hq, int, int, int) { return size_t(8) * B * Hq * T; }
int b200attn_bwd_mode(const void*, const void*, const void*, const void*, const float*, const void*, void*, void*, void*, int, int, int, int, int, int, float, int, void* ws, size_t n, void*) { return use(ws, n); }
size_t b200attn_decode_workspace_bytes(int B, int L, int Hq, int, int, int) { return size_t(4) * B * Hq * L; }
int b200attn_decode(const void*, const void*, const void*, void*, float*, int, int, int, int, int, float, int, void* ws, size_t n, void*) { return use(ws, n); }
int b200attn_decode_cached(const void*, const void*, const void*, void*, float*, int, int, int, int, int, int, float, int, void* ws, size_t n, void*) { return use(ws, n); }
size_t b200attn_rope_norm_bwd_workspace_bytes(int D) { return size_t(64) * D; }
int b200attn_rope_norm_fwd(const void*, int, int, void*, int, float*, const float*, const float*, const float*, int, int, int, int, float, void*) { return 0; }
int b200attn_rope_norm_bwd(const void*, int, const void*, int, int, const float*, const float*, const float*, const float*, void*, float*, int, int, int, int, void* ws, size_t n, void*) { return use(ws, n); }
int b200attn_kv_append(const void*, const void*, const void*, int, void*, void*, void*, const float*, const float*, const float*, const float*, int, int, int, int, int, int, int, float, void*) { return 0; }
const char* b200attn_strerror(int) { return ""; }
}
int main() {
    auto bf = [](std::int64_t n) { return Tensor({n}, DType::BF16, Device::Cuda); };
    auto backward = [&](void* stream, int T) {
        const int n = T * 64;
        Tensor q = bf(n), k = bf(n), v = bf(n), c = bf(n), d = bf(n), dq = bf(n), dk = bf(n), dv = bf(n), L({T}, DType::FP32, Device::Cuda);
        b200::flash_attn_backward(q, k, v, c, L, d, dq, dk, dv, 1, T, 64, 16, stream);
    };
    auto decode = [&](void* stream, int L) {
        Tensor q = bf(64), k = bf(L * 64), v = bf(L * 64), o = bf(64);
        b200::flash_attn_decode(q, k, v, o, 1, L, 1, 1, 64, stream);
    };
    void* s = reinterpret_cast<void*>(8);
    std::vector<std::thread> t;
    for (int i = 0; i < 4; ++i)
        t.emplace_back([&, i] {
            for (int r = 1; r <= 6; ++r) {
                backward(s, 128 * (1 + (r + i) % 5));  // of different sizes: the workspace grows while others use it
                backward(nullptr, 128);
                decode(s, 100 * r);
            }
        });
    for (auto& x : t) x.join();
    std::printf("%d calls, %d overlaps\n", calls.load(), overlaps.load());
    return overlaps.load() != 0;
}
"""


def test_calls_of_several_threads_never_share_a_workspace(tmp_path):
    (tmp_path / "core").mkdir()
    (tmp_path / "core" / "tensor.h").write_text(TENSOR)
    (tmp_path / "cuda_runtime.h").write_text("#pragma once\n#include <cstddef>\nenum { cudaSuccess = 0 };\nextern \"C\" int cudaGetDevice(int*);\n")
    (tmp_path / "harness.cc").write_text(HARNESS)
    exe = str(tmp_path / "harness")
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", f"-I{tmp_path}", f"-I{CSRC}", f"-I{os.path.join(ROOT, 'include')}",
                    str(tmp_path / "harness.cc"), os.path.join(CSRC, "modernllm_shim.cc"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("72 calls"), out.stdout + out.stderr

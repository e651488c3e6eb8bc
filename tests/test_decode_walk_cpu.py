"""The decode's early look at a ragged batch, run on the host: it reads the lengths while the kernel in front may still be writing
them, so the total, the place of a CTA's first tile and the walk on from there can each see other lengths.  Whatever they see, it
reads no length beyond the last sequence's and asks for no tile outside the cache."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "modern-llm-v1_b200", "csrc")

# The lengths end where a page without access begins.  The start of the walk (on the device a sum and a search over the lanes of
# a warp) is restated here: range from one set of lengths, sequence and tile from another.
DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <sys/mman.h>
#include <unistd.h>
#include "attn_decode.cuh"
using namespace b200attn;
template <int KEYS>
static int tiles_of(const DecodeParams& p, int b) { return (decode_len(p, b) + KEYS - 1) / KEYS; }
template <int KEYS>
static long run(std::mt19937& rng, int* end_of_page) {
    auto upto = [&](int lo, int hi) { return lo + int(rng() % unsigned(hi - lo + 1)); };
    DecodeParams p = {};
    p.B = upto(1, 70), p.units_per_seq = upto(1, 8), p.L = upto(1, 3000);
    int* lens = end_of_page - p.B;
    p.lens = lens;
    auto draw = [&](int kind) {
        for (int b = 0; b < p.B; ++b) lens[b] = kind == 0 ? upto(-5, p.L + 5) : kind == 1 ? upto(1, 1 + p.L / 8) : kind == 2 ? p.L : int(rng());
    };
    draw(upto(0, 3));
    DecodeWalk w = {};
    for (int b = 0; b < p.B; ++b) w.total += tiles_of<KEYS>(p, b) * p.units_per_seq;
    w.n_ctas = std::min(upto(1, 320), w.total);
    if (upto(0, 3)) draw(upto(0, 3));  // the kernel in front has written them
    long visits = 0;
    for (int c = 0; c < w.n_ctas; ++c) {
        DecodeWalk x = w;
        x.t = decode_range(w, c), x.t_end = decode_range(w, c + 1);
        x.b = p.B - 1, x.len = x.n_tiles = 1, x.u = x.j0 = 0;
        for (int b = 0, before = 0; b < p.B; before += tiles_of<KEYS>(p, b) * p.units_per_seq, ++b) {
            const int n = tiles_of<KEYS>(p, b);
            if (x.t >= before + n * p.units_per_seq) continue;
            x.b = b, x.len = decode_len(p, b), x.n_tiles = n;
            x.u = (x.t - before) / n, x.j0 = (x.t - before) % n;
            break;
        }
        if (upto(0, 7) == 0) draw(upto(0, 3));
        for (int left : {2, 1 << 20})
            decode_first_tiles<KEYS>(p, x, left, [&](int b, int u, int tile) {
                if (b < 0 || b >= p.B || u < 0 || u >= p.units_per_seq || tile < 0 || tile * KEYS >= p.L)
                    std::printf("outside: sequence %d of %d, unit %d, tile %d\n", b, p.B, u, tile), std::exit(1);
                ++visits;
            });
    }
    return visits;
}
int main() {
    const long page = sysconf(_SC_PAGESIZE);
    char* m = static_cast<char*>(mmap(nullptr, 2 * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (m == MAP_FAILED || mprotect(m + page, page, PROT_NONE)) return 2;
    std::mt19937 rng(5);
    long visits = 0;
    for (int i = 0; i < 4000; ++i)
        visits += i % 2 ? run<128>(rng, reinterpret_cast<int*>(m + page)) : run<64>(rng, reinterpret_cast<int*>(m + page));
    std::printf("%ld tiles\n", visits);
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("decode_walk")
    src, exe = d / "walk.cu", d / "walk"
    src.write_text(DRIVER)
    subprocess.check_call([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-I", CSRC,
                           "-o", str(exe), str(src)])
    return str(exe)


def test_early_look_stays_inside_the_lengths_and_the_cache(driver):
    r = subprocess.run([driver], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, f"exit {r.returncode}: {r.stdout[-300:]}"
    assert int(r.stdout.split()[0]) > 100000

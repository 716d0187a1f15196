"""Host code around the CUDA runtime, built against a stand-in runtime (tests/fake_cuda) and run here."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def _run(tmp_path, code):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    src = tmp_path / "t.cpp"
    src.write_text(code)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{ROOT / 'tests' / 'fake_cuda'}",
                    f"-I{ROOT / 'cupyram_b200' / 'csrc'}", str(src), "-o", str(tmp_path / "t")], check=True)
    return subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=120)


def test_staged_copies_are_whole_and_stay_on_their_device(tmp_path):
    """Copies of a piece less, a piece more and several rings, on device 3, from a thread whose
    current device that is: the bytes arrive, and no call - the copying threads' included - is
    made with another device current."""
    r = _run(tmp_path, r"""
#include "staging.h"
#include <cstdio>
#include <vector>
int main() {
    cudaSetDevice(3);
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    const size_t sizes[] = {crk::kOutMin, crk::kOutMin + 1, 3 * crk::kOutPiece - 7, 2 * crk::kStageChunk,
                            2 * crk::kStageChunk + 5, 5 * crk::kStageChunk + 12345};
    for (size_t n : sizes) {
        std::vector<unsigned char> a(n), b(n + 8, 0xee), c(n + 8, 0xee);
        for (size_t i = 0; i < n; ++i) a[i] = (unsigned char)(i * 2654435761u >> 13);
        if (crk::staged_h2d(3, b.data(), a.data(), n, st) != cudaSuccess) return 1;
        if (crk::staged_d2h(3, c.data(), b.data(), n, st) != cudaSuccess) return 2;
        if (memcmp(a.data(), c.data(), n) || c[n] != 0xee) return printf("size %zu differs\n", n), 3;
    }
    if (fake::wrong_device) return printf("%d calls on another device\n", fake::wrong_device), 4;
    return 0;
}
""")
    assert r.returncode == 0, r.stdout + r.stderr


def test_lanes_are_idle_when_they_are_taken_again(tmp_path):
    """A lane given back with work still on it (an engine whose march failed between its
    launches) is not handed on before that work is done; the pool keeps a bounded number
    per device, hands out a device's own, and clear destroys them."""
    r = _run(tmp_path, r"""
#include "lanes.h"
#include <cstdio>
int main() {
    crk::LanePool pool;
    crk::StreamLane l, m;
    char a[4] = "abc", b[4] = "";
    cudaSetDevice(2);
    if (pool.take(2, &l) != cudaSuccess) return 1;
    cudaMemcpyAsync(b, a, 4, cudaMemcpyHostToDevice, l.stream);  // never waited for
    pool.give(2, l);
    if (pool.take(2, &m) != cudaSuccess || m.stream != l.stream) return 2;
    if (!m.stream->work.empty() || b[0] != 'a') return printf("a busy lane was handed on\n"), 3;
    pool.give(2, m);
    cudaSetDevice(1);
    if (pool.take(1, &l) != cudaSuccess || l.stream == m.stream || l.stream->device != 1) return 4;
    std::vector<crk::StreamLane> many(crk::LanePool::kKept + 20);
    for (auto& x : many) pool.take(1, &x);
    for (auto& x : many) pool.give(1, x);
    pool.give(1, l);
    if (fake::streams_alive != (int)crk::LanePool::kKept + 1) return 5;
    pool.clear();
    if (fake::streams_alive) return 6;
    return 0;
}
""")
    assert r.returncode == 0, r.stdout + r.stderr

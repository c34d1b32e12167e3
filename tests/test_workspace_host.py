"""The scratch pool (csrc/workspace_pool.h) against an allocator that runs out, built for the host: what a growth that fails leaves behind."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "workspace_pool.h"

#include <cstdio>

#define EXPECT(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    const size_t MB = size_t{1} << 20;
    atoma::WorkspacePool pool;
    const atoma::WorkspacePool::Key a(0, 5, nullptr), b(0, 6, nullptr);
    size_t room = 40 * MB;
    int calls = 0;
    char *next = reinterpret_cast<char *>(0x1000);
    auto alloc = [&](size_t n) -> void * {
        ++calls;
        if (n > room) return nullptr;
        room -= n;
        next += n;
        return next;
    };
    int asked = 0;
    auto yes = [&] { ++asked; return true; };
    auto no = [&] { ++asked; return false; };
    void *first = pool.get(a, 9 * MB + 1, yes, alloc);
    EXPECT(first && room == 30 * MB);
    EXPECT(asked == 1);
    EXPECT(pool.get(a, 10 * MB, yes, alloc) == first && calls == 1 && asked == 1);       // rounded up to whole MiB; a block that fits asks nothing
    // a growth that fails: the block that was there still serves what fits it, and nothing was lost
    EXPECT(pool.get(a, 31 * MB, yes, alloc) == nullptr && room == 30 * MB);
    EXPECT(pool.get(a, 10 * MB, yes, alloc) == first && room == 30 * MB);
    for (int i = 0; i < 100; ++i) {
        EXPECT(pool.get(a, 31 * MB, yes, alloc) == nullptr);
        EXPECT(pool.get(a, 5 * MB, yes, alloc) == first);
    }
    EXPECT(room == 30 * MB);
    // not allowed to grow (a stream that is being captured): the block as it is, or none; the allocator is not asked
    calls = 0;
    EXPECT(pool.get(a, 10 * MB, no, alloc) == first && pool.get(a, 11 * MB, no, alloc) == nullptr && pool.get(b, 1, no, alloc) == nullptr && calls == 0);
    // a growth is by half at least, so that many small ones do not set many blocks aside; where that is too much, what is asked for
    EXPECT(pool.get(a, 10 * MB + 1, yes, alloc) != first && room == 15 * MB);
    EXPECT(pool.get(a, 15 * MB, yes, alloc) != nullptr && room == 15 * MB);
    EXPECT(pool.get(b, 6 * MB, yes, alloc) != nullptr && room == 9 * MB);
    EXPECT(pool.get(b, 8 * MB, yes, alloc) != nullptr && room == 0);
    room = 8 * MB + MB / 2;
    EXPECT(pool.get(b, 9 * MB + 1, yes, alloc) == nullptr && pool.get(b, 9 * MB, yes, alloc) != nullptr && room == 8 * MB + MB / 2);
    std::printf("ok\n");
    return 0;
}
"""


def test_a_growth_that_fails_leaves_the_block_in_service(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'atoma_infer_b200' / 'csrc'}", str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout

"""Which host buffers a kernel is given where they are (host_range.hpp), with a fake of the lookup of a byte's mapping."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WALK = r"""
#include <cstdio>
#include <initializer_list>
#include "host_range.hpp"
// Pages 16 .. 19 and 21 .. 31 are pinned, 20 is not.
static int asked = 0;
static bool mapped(const void* p) {
    const uintptr_t page = reinterpret_cast<uintptr_t>(p) / 4096;
    ++asked;
    return page >= 16 && page < 32 && page != 20;
}
static int bad = 0;
static void expect(bool want, size_t first, size_t bytes) {
    asked = 0;
    if (hc::host_range_mapped(mapped, reinterpret_cast<const void*>(first), bytes) == want && asked <= int(bytes / 4096) + 3) return;
    std::printf("%zu bytes at %zu: not %d, or asked %d times\n", bytes, first, int(want), asked);
    ++bad;
}
int main() {
    const size_t page = 4096;
    for (size_t bytes : {size_t(16), size_t(4080), page, page + 16, 2 * page + 64, 4 * page}) {
        expect(true, 16 * page, bytes);                     // from the start of what is pinned
        expect(true, 20 * page - bytes, bytes);             // up to its end
        expect(true, 32 * page - bytes, bytes);
        expect(false, 20 * page - bytes + 16, bytes);       // 16 bytes past it
        expect(false, 32 * page - bytes + 16, bytes);
        expect(false, 16 * page - 16, bytes + 16);          // 16 bytes before it
    }
    expect(false, 18 * page, 8 * page);                     // both ends pinned, a page between them is not
    expect(false, 19 * page + 4080, page + 32);
    expect(true, 21 * page, 11 * page);
    expect(false, 16 * page, 0);
    return bad != 0;
}
"""


def test_buffers_pinned_in_part_are_not_for_a_kernel(tmp_path):
    (tmp_path / "walk.cpp").write_text(WALK)
    program = str(tmp_path / "walk")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "hydra_b200", "csrc"), str(tmp_path / "walk.cpp"), "-o", program])
    done = subprocess.run([program], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout

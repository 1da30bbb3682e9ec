"""The bookkeeping of a request server lane's memory (csrc/pa_arena.h): pieces never
overlap and stay inside the range, whatever the order they come back in, and all of
them together make up the whole range again."""
import os
import subprocess

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "pa_arena.h"
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main()
{
    struct Piece { uint64_t at, len; };
    const uint64_t none = pa::Arena::kNone, A = pa::Arena::kAlign;
    const uint64_t totals[] = {A, 9 * A, 1 << 20, ((uint64_t)1 << 34) + 7 * A};
    for (uint64_t total : totals) {
        pa::Arena a;
        CHECK(a.take(1) == none && !a.give(0));    // nothing to hand out yet
        a.add(0, total);
        CHECK(a.take(0) == none && a.take(total + 1) == none && a.take(~0ull) == none && !a.give(0));
        std::srand((unsigned)total);
        std::vector<Piece> held;
        for (int step = 0; step < 20000; ++step) {
            if (std::rand() % 2) {
                const uint64_t len = 1 + (uint64_t)std::rand() % (total / (1 + std::rand() % 40) + 1);
                const uint64_t at = a.take(len);
                if (at == none) continue;
                CHECK(at + len <= total && at % A == 0);
                for (const Piece &q : held) CHECK(at + len <= q.at || q.at + q.len <= at);
                held.push_back({at, len});
            } else if (!held.empty()) {
                const size_t i = std::rand() % held.size();
                CHECK(!a.give(held[i].at + 1));
                CHECK(a.give(held[i].at) && !a.give(held[i].at));
                held.erase(held.begin() + i);
            }
        }
        for (const Piece &q : held) CHECK(a.give(q.at));
        CHECK(a.pieces().size() == 1 && a.take(total) == 0);   // one piece again
        CHECK(a.take(1) == none && a.give(0) && !a.give(total));
        // cut out of the front, the middle and the end, and put back
        for (uint64_t at : {(uint64_t)0, total / 2 / A * A, total - A}) {
            a.cut(at, A);
            uint64_t left = 0;
            for (const auto &f : a.pieces()) {
                CHECK(f.first + f.second <= at || f.first >= at + A);
                left += f.second;
            }
            CHECK(left == total - A);
            a.add(at, A);
            CHECK(a.pieces().size() == 1 && a.pieces().begin()->second == total);
        }
    }
    return 0;
}
"""


def test_arena_pieces(tmp_path):
    csrc = os.path.join(os.path.dirname(__file__), "..", "cuppa-public_b200", "csrc")
    src, exe = tmp_path / "arena.cpp", tmp_path / "arena"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-fsanitize=undefined",
                    "-I", csrc, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

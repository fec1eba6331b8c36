"""Buffers that are replaced together (csrc/buffer_set.cuh): whichever allocation fails, no pointer outlives its buffer, nothing leaks and the
next attempt starts over.  Compiled for the host with an allocator that fails on demand."""
import subprocess
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "nano-inference_b200" / "csrc"

PROGRAM = r"""
#include "buffer_set.cuh"
#include <cstdio>
#include <cstdlib>
#include <set>

static std::set<void*> live;
static int until_failure = -1;
static bool alloc(void** p, size_t n) {
    if (until_failure-- == 0) return false;
    *p = std::malloc(n); live.insert(*p); return true;
}
static void free_one(void* p) { if (!live.erase(p)) { std::printf("freed twice\n"); std::exit(1); } std::free(p); }
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

struct Owner { float* a = nullptr; double* b = nullptr; struct { unsigned* q; double* d; } t{}; mi::BufferSet mem; };
static bool fill(Owner& o, size_t n) {
    return o.mem.take(&o.a, 4 * n, alloc) && o.mem.take(&o.b, 8 * n, alloc) && o.mem.take(&o.t.q, 4 * n, alloc) && o.mem.take(&o.t.d, 8 * n, alloc);
}
int main() {
    for (int k = 0; k <= 4; k++) {
        Owner o;
        until_failure = -1;
        CHECK(fill(o, 8) && live.size() == 4);
        o.mem.release(free_one);                                    // larger ones are wanted ..
        CHECK(!o.a && !o.b && !o.t.q && !o.t.d && live.empty());
        until_failure = k;
        const bool ok = fill(o, 16);                                // .. and the k-th of them is refused
        CHECK(ok == (k == 4) && live.size() == (size_t)k);
        CHECK(!o.a == (k < 1) && !o.b == (k < 2) && !o.t.q == (k < 3) && !o.t.d == (k < 4));
        for (void* p : {(void*)o.a, (void*)o.b, (void*)o.t.q, (void*)o.t.d}) CHECK(!p || live.count(p));
        o.mem.release(free_one);
        CHECK(!o.a && !o.b && !o.t.q && !o.t.d && live.empty());
        until_failure = -1;
        CHECK(fill(o, 8) && live.size() == 4);
        o.mem.release(free_one);
        CHECK(live.empty());
    }
    return 0;
}
"""


def test_no_pointer_outlives_its_buffer(tmp_path):
    src = tmp_path / "bufs.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "bufs"
    subprocess.run(["g++", "-O2", "-Wall", "-std=c++17", "-I", str(SRC), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_the_m_token_buffers_are_such_a_set():
    """Every pointer of the M-token step is taken from the set, and released through it on every way out of the growth."""
    import re
    text = re.sub(r"//[^\n]*", "", (SRC / "verify.cu").read_text())
    body = text[text.index("int ensure_bufs("):text.index("void mi::free_verify_bufs")]
    assert "b.mem.take(" in body
    assert body.index("release_bufs(b)") < body.index("take(&b.X") < body.rindex("release_bufs(b)") < body.index("b.cap = cap")
    model = (SRC / "model.cuh").read_text()
    pointers = set(re.findall(r"\* (\w+) = nullptr;", model[model.index("struct VerifyBufs"):model.index("struct mi_model")])) - {"h_meta"}
    assert pointers and all(f"take(&b.{p}," in body for p in pointers), pointers

"""Device buffers and the context's scratch (engine.cuh: DBuf, Context::scratch_take) when the
device runs out of memory, with cudaMalloc faked: the call that asked gets LSJK_ENOMEM, and
later calls that fit get memory that is there."""
import ctypes

import pytest

from host_code import compile_host, source_part

FAKE = """
#include <atomic>
#include <cstdint>
#include <functional>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>
using cudaError_t = int;
using cudaStream_t = int;
constexpr int cudaSuccess = 0, cudaMemcpyHostToDevice = 1, LSJK_ENOMEM = 3;
long room, given;
int last_error;
std::vector<std::pair<char*, size_t>> live;
template <typename T> int cudaMalloc(T** p, size_t n)
{
    if (given + (long) n > room) return last_error = 2;   // (*p is left as it was)
    static uintptr_t next = 1 << 20;   // addresses only: nothing reads or writes there
    *p = (T*) next;
    next += n;
    live.push_back({(char*) *p, n});
    given += n;
    return 0;
}
int cudaFree(void* p)
{
    for (size_t k = 0; k < live.size(); ++k)
        if (live[k].first == p) { given -= live[k].second; live.erase(live.begin() + k); return 0; }
    return last_error = 1;
}
int cudaGetLastError() { const int e = last_error; last_error = 0; return e; }
const char* cudaGetErrorString(int) { return "fake"; }
int cudaMemcpyAsync(void*, const void*, size_t, int, cudaStream_t) { return 0; }
#define LSJK_CUDA(x) do { if ((x) != cudaSuccess) throw std::runtime_error(#x); } while (0)
struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};
std::atomic<long> g_device_allocations{0};
"""

CONTEXT = """
struct Context {
    std::vector<std::unique_ptr<DBuf<char>>> scratch;
    size_t scratch_used = 0;
    bool scratch_fixed = false;
    char* scratch_take(size_t bytes);
    bool scratch_take_all(size_t bytes, int count, char** out);
    void scratch_reset() { scratch_used = 0; }
};
"""

RUN = """
Context* c;
extern "C" void start(long r) { delete c; c = new Context; room = r; last_error = 0; }
extern "C" void reset() { c->scratch_reset(); }
extern "C" long held() { return given; }
// 1: memory that is there, all of it; 0: refused with LSJK_ENOMEM; below 0: something else
extern "C" int take(long bytes)
{
    try {
        char* p = c->scratch_take(bytes);
        if (cudaGetLastError()) return -1;
        for (auto& q : live)
            if (p >= q.first && p + bytes <= q.first + q.second) return 1;
        return -2;
    } catch (const Error& e) {
        return e.code != LSJK_ENOMEM ? -3 : (cudaGetLastError() ? -4 : 0);
    }
}
// 1: all of them, apart from one another; 0: none, and the scratch as it was
extern "C" int take_all(long bytes, int count)
{
    std::vector<char*> p(count);
    const size_t used = c->scratch_used;
    const long before = given;
    if (!c->scratch_take_all(bytes, count, p.data()))
        return used == c->scratch_used && given == before && !cudaGetLastError() ? 0 : -1;
    for (int k = 0; k < count; ++k) {
        bool there = false;
        for (auto& q : live) there = there || (p[k] >= q.first && p[k] + bytes <= q.first + q.second);
        if (!there) return -2;
        for (int j = 0; j < k; ++j)
            if (p[k] < p[j] + bytes && p[j] < p[k] + bytes) return -3;
    }
    return 1;
}
"""


def build(tmp_path, extra=""):
    parts = [source_part("engine.cuh", "template <typename T>\nstruct DBuf {", "// The arrays of one object as slices"),
             source_part("engine.cuh", "// Stream-ordered scratch: a bump allocator", "// The auxiliary streams of one build")]
    return compile_host(tmp_path, FAKE + parts[0] + CONTEXT + parts[1] + RUN + extra)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return build(tmp_path_factory.mktemp("scratch"))


MB = 1 << 20


def test_calls_after_a_refused_one(lib):
    L = ctypes.c_long
    lib.held.restype = L
    lib.start(L(300 * MB))
    assert lib.take(L(100 * MB)) == 1
    assert lib.take(L(500 * MB)) == 0          # no room
    for _ in range(2):                         # the next calls
        lib.reset()
        assert lib.take(L(90 * MB)) == 1
        assert lib.take(L(80 * MB)) == 1       # beyond the block there is
        assert lib.take(L(400 * MB)) == 0
    lib.reset()
    assert lib.take(L(300 * MB)) == 0
    lib.reset()
    assert [lib.take(L(60 * MB)) for _ in range(3)] == [1, 1, 1]
    assert lib.held() <= 300 * MB


def test_all_or_none(lib):
    L = ctypes.c_long
    lib.start(L(300 * MB))
    assert lib.take(L(70 * MB)) == 1
    assert lib.take_all(L(50 * MB), 3) == 1
    assert lib.take_all(L(30 * MB), 3) == 0
    assert lib.take(L(14 * MB)) == 1           # the rest of a block is still there
    lib.reset()
    assert lib.take_all(L(50 * MB), 4) == 1
    assert lib.take_all(L(100 * MB), 3) == 0

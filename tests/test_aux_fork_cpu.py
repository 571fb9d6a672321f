"""A build that throws between the fork to the auxiliary streams and the join still makes the
main stream wait for what was launched (engine.cuh: AuxFork), with the CUDA calls faked."""
import ctypes

import pytest

from host_code import compile_host, source_part

FAKE = """
#include <string>
#include <stdexcept>
// an event holds how much of each stream had been enqueued when it was recorded
using cudaStream_t = int;
using cudaEvent_t = int;
constexpr int cudaSuccess = 0;
constexpr int kStreams = 17;
int enqueued[kStreams], seen[kStreams][kStreams], event_seen[64][kStreams], calls, fail_at;
int call() { return ++calls == fail_at; }
int cudaEventRecord(int ev, int s)
{
    if (call()) return 1;
    for (int k = 0; k < kStreams; ++k) event_seen[ev][k] = k == s ? enqueued[s] : seen[s][k];
    return 0;
}
int cudaStreamWaitEvent(int s, int ev, int)
{
    if (call()) return 1;
    for (int k = 0; k < kStreams; ++k) seen[s][k] = seen[s][k] > event_seen[ev][k] ? seen[s][k] : event_seen[ev][k];
    return 0;
}
#define LSJK_CUDA(x) do { if ((x) != cudaSuccess) throw std::runtime_error(#x); } while (0)
struct Context {
    static constexpr int kAux = 16;
    int naux = kAux, stream = 0, aux[kAux], fork_ev = 0, join_ev[kAux];
    Context() { for (int i = 0; i < kAux; ++i) aux[i] = join_ev[i] = i + 1; }
};
"""

RUN = """
// launches on `used` streams, throws after them (or in the fail-th CUDA call); 1 if an
// exception came out, 2 if the main stream does not then wait for every launch
extern "C" int run(long npair, int used, int throws, int fail)
{
    Context c;
    calls = 0;
    fail_at = fail;
    for (int i = 0; i < kStreams; ++i) {
        enqueued[i] = 0;
        for (int k = 0; k < kStreams; ++k) seen[i][k] = 0;
    }
    enqueued[0] = 1;
    int rc = 0;
    try {
        AuxFork fork(&c, npair);
        for (int i = 0; i < used; ++i) {
            OnAux on(&c, i);
            if (seen[c.stream][0] != 1) rc |= 4;   // launched before the main stream's work
            ++enqueued[c.stream];
            if (throws && i + 1 == used) throw std::runtime_error("launch");
        }
        fork.join();
    } catch (const std::runtime_error&) {
        rc |= 1;
    }
    if (c.stream != 0) rc |= 8;
    for (int i = 1; i < kStreams; ++i)
        if (seen[0][i] != enqueued[i]) rc |= 2;
    return rc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    part = source_part("engine.cuh", "// The auxiliary streams of one build", "template <typename T>\ninline T* take(")
    return compile_host(tmp_path_factory.mktemp("fork"), FAKE + part + RUN)


@pytest.mark.parametrize("npair", [100, 100000])
@pytest.mark.parametrize("used", [1, 5, 40])
def test_join_on_every_way_out(lib, npair, used):
    run = lambda *a: lib.run(ctypes.c_long(npair), used, *a)
    assert run(0, 0) == 0
    assert run(1, 0) == 1
    n = 8 if npair < 20000 else 16
    for fail in (n + 2, n + 5, 3 * n + 1):   # an error of a call of the join itself: it is tried again
        assert run(0, fail) == 1

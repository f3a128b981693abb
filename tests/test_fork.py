"""The side streams of a stage (csrc/fork.h), compiled here against a stand-in
for the CUDA runtime that writes down each call: they have the priority of the
caller's stream, a stream of an SM partition gets none, a stage that ends
early on an error still makes the caller's stream wait for their work, and the
pool of idle ones is bounded."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "cgfdm-fp16_sve_sme_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <cstdio>
struct FakeStream { const char *name; int prio; bool part, broken; };
struct FakeEvent { int id; };
typedef FakeStream *cudaStream_t;
typedef FakeEvent *cudaEvent_t;
enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 999 };
enum { cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1 };
inline int g_streams, g_events, g_live, g_fail_wait = -1;
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = new FakeEvent{g_events++}; ++g_live; return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; --g_live; return cudaSuccess; }
inline cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int p) {
  static char names[400][8];
  std::snprintf(names[g_streams], sizeof names[0], "s%d", g_streams);
  *s = new FakeStream{names[g_streams++], p, false, false}; ++g_live; return cudaSuccess;
}
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { delete s; --g_live; return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  return s->broken ? cudaErrorUnknown : cudaSuccess;
}
inline cudaError_t cudaStreamGetPriority(cudaStream_t s, int *p) { *p = s->prio; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::printf("record %d on %s\n", e->id, s->name); return cudaSuccess;
}
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (g_fail_wait == e->id) return cudaErrorUnknown;
  std::printf("%s waits for %d\n", s->name, e->id); return cudaSuccess;
}
"""

MAIN = r"""
#include <initializer_list>
#include "fork.h"
namespace cgfdm { bool stream_is_partitioned(cudaStream_t st) { return st->part; } }
using namespace cgfdm;
static int stage(Fork &f, cudaStream_t st, bool fails, bool in_turn = false) {
  Branches br(f, st, in_turn);
  if (br.begin() != cudaSuccess) return 1;
  std::printf("launch on %s %s\n", br.side(0)->name, br.side(1)->name);
  if (fails) return 1;
  return br.join() == cudaSuccess ? 0 : 1;
}
int main() {
  FakeStream a{"a", 0, false, false}, high{"high", -5, false, false}, part{"part", 0, true, false};
  Fork f;
  for (cudaStream_t st : {&a, &high, &part, &a}) {
    std::printf("# %s\n", st->name);
    if (f.attach(0, st) != cudaSuccess) return 1;
    if (f.set()) std::printf("priorities %d %d\n", f.set()->side[0]->prio, f.set()->side[1]->prio);
    stage(f, st, false);
  }
  std::printf("# fails\n");
  std::printf("rc %d\n", stage(f, &a, true));
  std::printf("# in turn\n");
  stage(f, &a, false, true);
  std::printf("# branch refused\n");
  g_fail_wait = f.set()->start->id;
  std::printf("rc %d\n", stage(f, &a, false));
  g_fail_wait = -1;
  f.destroy();
  std::printf("# pooled %d\n", g_live);
  Fork h, other;
  h.attach(0, &high);
  other.attach(1, &a);
  std::printf("# next owner %s, another device %s\n", h.set()->side[0]->name,
              other.set()->side[0]->name);
  h.set()->side[1]->broken = true;
  h.destroy();
  other.destroy();
  std::printf("# after an error %d\n", g_live);
  static Fork many[40];
  for (Fork &m : many) m.attach(0, &a);
  for (Fork &m : many) m.destroy();
  std::printf("# at most %d\n", g_live);
}
"""


@pytest.fixture(scope="module")
def said(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = str(tmp_path_factory.mktemp("fork"))
    with open(os.path.join(d, "cuda_runtime.h"), "w") as f:
        f.write(RUNTIME)
    with open(os.path.join(d, "main.cpp"), "w") as f:
        f.write(MAIN)
    exe = os.path.join(d, "main")
    subprocess.check_call([cxx, "-std=c++17", "-I", d, "-I", CSRC, os.path.join(d, "main.cpp"),
                           "-o", exe])
    parts = {}
    for line in subprocess.check_output([exe], text=True).splitlines():
        if line.startswith("# "):
            parts.setdefault(line[2:], []).append([])
            last = parts[line[2:]][-1]
        else:
            last.append(line)
    return parts


def _joined(lines, st, sides):
    """Every side stream waits for an event of st first, and st for one of each last."""
    rec = {l.split()[1]: l.split()[3] for l in lines if l.startswith("record")}
    wait = [(l.split()[0], rec[l.split()[3]]) for l in lines if "waits for" in l]
    assert wait == [(s, st) for s in sides] + [(st, s) for s in sides]


def test_side_streams_have_the_callers_priority(said):
    first, again = said["a"]
    assert "priorities 0 0" in first and "launch on s0 s1" in first
    assert "priorities -5 -5" in said["high"][0] and "launch on s2 s3" in said["high"][0]
    _joined(first, "a", ["s0", "s1"])
    _joined(said["high"][0], "high", ["s2", "s3"])
    assert again == first  # the set of that priority again


def test_a_partitioned_stream_runs_in_turn(said):
    assert said["part"][0] == ["launch on part part"]
    assert said["in turn"][0] == ["launch on a a"]


def test_a_failing_stage_joins_its_branches(said):
    lines = said["fails"][0]
    assert lines[-1] == "rc 1"
    _joined(lines, "a", ["s0", "s1"])
    assert said["branch refused"][0][-1] == "rc 1"


def test_idle_sets_go_to_the_next_owner_of_the_device(said):
    """Five streams and events a set; at most 32 sets are kept, none that an
    error left behind, and none for another device or priority."""
    assert "pooled 10" in said and "next owner s2, another device s4" in said
    assert "after an error 10" in said  # the broken set went, the other device's stays
    assert "at most %d" % (32 * 5) in said

"""Host tables and the asynchronous copies that read them
(csrc/hosttables.cuh), against a CUDA runtime whose copies read the host
memory only when they are waited for, as a copy from pageable memory may."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mpi-rockstar_gb300", "csrc")

PROGRAM = r"""
#include <stdio.h>
#include <string.h>
#include <vector>
#include <stdexcept>
#include "hosttables.cuh"

struct Copy { void *d; const void *s; size_t n; };
static std::vector<Copy> queued;
static size_t marked = 0;  // copies before the event's last record
static int fail_create = 0, fail_copy = 0, fail_record = 0, live = 0, syncs = 0;
static void drain(size_t k) {
    for (size_t i = 0; i < k && i < queued.size(); i++) memcpy(queued[i].d, queued[i].s, queued[i].n);
    queued.erase(queued.begin(), queued.begin() + (k < queued.size() ? k : queued.size()));
}
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    if (fail_create) return cudaErrorMemoryAllocation;
    *e = (cudaEvent_t)&live;
    live++;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { live--; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) {
    if (fail_record) return cudaErrorUnknown;
    marked = queued.size();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { syncs++; drain(marked); marked = 0; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { syncs++; drain(queued.size()); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fail_copy) return cudaErrorUnknown;
    queued.push_back(Copy{d, s, n});
    return cudaSuccess;
}
}
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

static std::vector<int> numbers(int n, int first) {
    std::vector<int> v(n);
    for (int i = 0; i < n; i++) v[i] = first + i;
    return v;
}
static void churn() {  // what frees here is written over
    for (int k = 0; k < 64; k++) { std::vector<int> x(1000 + k, -1); asm volatile("" ::"r"(x.data()) : "memory"); }
}
int main() {
    std::vector<int> a(1000), b(1007), c(1003);
    {
        rsg::HostTables t(0);
        {
            std::vector<int> x = numbers(1000, 5), y = numbers(1007, 70);
            CHECK(t.copy(a.data(), std::move(x)) == cudaSuccess);
            CHECK(t.copy(b.data(), std::move(y)) == cudaSuccess);
            CHECK(t.copy(c.data(), numbers(0, 0)) == cudaSuccess);  // empty: no copy
            CHECK(t.copy(c.data(), numbers(1003, 9)) == cudaSuccess);
        }
        churn();
        CHECK(queued.size() == 3 && syncs == 0);
    }
    CHECK(a == numbers(1000, 5) && b == numbers(1007, 70) && c == numbers(1003, 9));
    CHECK(queued.empty() && live == 0 && syncs == 1);
    try {  // an error unwinds the caller
        rsg::HostTables t(0);
        t.copy(a.data(), numbers(1000, 40));
        throw std::runtime_error("");
    } catch (std::runtime_error &) {
    }
    CHECK(a == numbers(1000, 40) && live == 0);
    { rsg::HostTables t(0); }  // nothing copied: nothing waited for
    CHECK(syncs == 2);
    fail_create = 1;
    { rsg::HostTables t(0); CHECK(t.copy(a.data(), numbers(1000, 1)) != cudaSuccess); }
    CHECK(queued.empty());
    fail_create = 0;
    fail_copy = 1;
    { rsg::HostTables t(0); CHECK(t.copy(a.data(), numbers(1000, 1)) != cudaSuccess); }
    CHECK(live == 0);
    fail_copy = 0;
    fail_record = 1;  // the copy is out: it is waited for at once
    { rsg::HostTables t(0); CHECK(t.copy(a.data(), numbers(1000, 3)) != cudaSuccess); CHECK(queued.empty()); }
    CHECK(a == numbers(1000, 3) && live == 0);
    printf("ok\n");
    return 0;
}
"""


def cuda_include():
    from conftest import load_pkg
    load_pkg()
    import mpi_rockstar_gb300.builder as b
    nvcc = b._nvcc()
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def test_tables_live_until_their_copies_are_done(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", cuda_include(), str(src),
                           "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout


@pytest.mark.gpu
def test_sorts_and_potentials_in_a_row(rk):
    """Small segments only (no count is read back after their tables are
    sent) and nodes of the block and chunked forms, call after call: the
    same bytes every time."""
    import numpy as np
    p, box, mp, _ = rk.synth(1, 0.1)
    cfg = rk.Config(particle_mass=mp, box_size=box, total_particles=len(p))
    fp, off, sz = rk.rockstar_fof(p, cfg)
    rng = np.random.default_rng(0)
    po = np.zeros(150000, rk.POTENTIAL)
    po["pos"][:, :3] = 20 + rng.normal(size=(len(po), 3))
    first = {}
    for k in range(12):
        q, h, e = rk.find_subs(fp, off, sz, cfg, batched=bool(k & 1))
        e["_pad"] = 0  # the record's padding, which nothing writes
        pe = rk.compute_potential(po, cfg, form=1)["pe"]
        for name, got in ((k & 1, q.tobytes() + h.tobytes() + e.tobytes()), ("pe", pe.tobytes())):
            assert first.setdefault(name, got) == got

"""The meetings of the cooperative launches (ring order, compaction): a wait
that runs out ends the launch with an error, on the main sequence also with the
halt, before anything that the other blocks would have written is used; the
launches after it do nothing.  Their grids are no larger than the device holds at
once, and a launch that it refuses is reported.  The kernels are compiled here with a short limit
and launched as one block that is told to wait for arrivals that never come."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include "k_topology.cu"
#include <cstring>
namespace lbib {
void launch_clear_forces(MembraneDev&, cudaStream_t, const Status*) {}
}
using namespace lbib;

// One launch of one block over a membrane without nodes; `missing`: arrivals
// that it waits for in vain.  out: the error and, if it was raised beside the main
// sequence, its stage, halt, haltStage, changed, removed, a wait ran out,
// ringStart[0]; then the error and `changed` after a second launch whose status
// word is clear.
static int error_of(const Status& s) { return s.beside ? 255 - (int)((s.beside >> 32) & 255) : s.err; }
extern "C" int meet(int compaction, int beside, unsigned missing, int* out) {
    const int n = 64;
    int* a;
    if (cudaMalloc(&a, 32 * n * sizeof(int)) != cudaSuccess) return 1;
    cudaMemset(a, 0, 32 * n * sizeof(int));
    auto part = [&](int k) { return a + k * n; };
    Topo tp{};
    tp.changed = 1;
    tp.removed = 1;
    Status s{};
    unsigned meetings[3] = {0u, missing, 0u};
    int five = 5;
    MembraneDev m{};
    m.topo = (Topo*)part(0);
    m.Mcap = m.Ccap = n;
    m.nCells = 1;
    m.ca = part(1); m.cb = part(2); m.next = part(3); m.prev = part(4); m.ringStart = part(5); m.ringNode = part(6);
    m.cdom = (uint32_t*)part(7); m.id = (uint32_t*)part(8);
    TopoDev t{};
    t.cellCount = part(9); t.cellFill = part(10); t.cellStart = part(11); t.outConn = part(12);
    t.firstConn = part(13); t.cellOfDom = part(14); t.members = part(15); t.succ = part(16); t.dist = part(17);
    t.blockSum = part(18); t.rank = part(19); t.nrank = part(20); t.ringMeet = (unsigned*)part(21);
    t.nDomains = 1;
    t.nCellsCap = 1;
    Status* st = (Status*)part(24);
    cudaMemcpy(m.topo, &tp, sizeof tp, cudaMemcpyHostToDevice);
    cudaMemcpy(st, &s, sizeof s, cudaMemcpyHostToDevice);
    cudaMemcpy(t.ringMeet, meetings, sizeof meetings, cudaMemcpyHostToDevice);
    cudaMemcpy(m.ringStart, &five, sizeof five, cudaMemcpyHostToDevice);
    for (int launch = 0; launch < 2; ++launch) {
        if (compaction) coarsen_compact_kernel<<<1, 256>>>(m, t, 0, st, 0);
        else rings_kernel<<<1, 256>>>(m, t, 1, st, beside);
        if (cudaDeviceSynchronize() != cudaSuccess || cudaGetLastError() != cudaSuccess) return 2;
        cudaMemcpy(&s, st, sizeof s, cudaMemcpyDeviceToHost);
        cudaMemcpy(&tp, m.topo, sizeof tp, cudaMemcpyDeviceToHost);
        if (launch == 1) break;
        cudaMemcpy(meetings, t.ringMeet, sizeof meetings, cudaMemcpyDeviceToHost);
        cudaMemcpy(&five, m.ringStart, sizeof five, cudaMemcpyDeviceToHost);
        const int got[8] = {error_of(s), s.beside ? beside_stage(s.beside) : 0, s.halt, s.haltStage, tp.changed, tp.removed, (int)meetings[2], five};
        std::memcpy(out, got, sizeof got);
        std::memset(&s, 0, sizeof s);
        cudaMemcpy(st, &s, sizeof s, cudaMemcpyHostToDevice);
    }
    out[8] = error_of(s);
    out[9] = tp.changed;
    cudaFree(a);
    return 0;
}

// The error of a ring launch over a membrane of 2^24 nodes, unchanged since its
// last ranking (every block returns at once), on a grid of at most `blocks`
// (0: meet_blocks).  *most: meet_blocks.
extern "C" int grid(int blocks, int* most) {
    if (meet_blocks(most) != cudaSuccess) return -1;
    int* a;
    if (cudaMalloc(&a, 4096) != cudaSuccess) return -1;
    cudaMemset(a, 0, 4096);
    MembraneDev m{};
    m.topo = (Topo*)a;
    m.Mcap = m.Ccap = 1 << 24;
    TopoDev t{};
    t.nCellsCap = 1;
    t.meetBlocks = blocks ? blocks : *most;
    t.ringMeet = (unsigned*)(a + 512);
    launch_rings(m, t, (Status*)(a + 256), 0);
    const int e = (int)cudaGetLastError();
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    cudaFree(a);
    return e;
}
"""
ERR_STATE, ST_COARSEN, ST_BIO = 91, 11, 13


@pytest.fixture(scope="module")
def meet(tmp_path_factory):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lbibcell_b200 import build
    where = tmp_path_factory.mktemp("meeting")
    source, library = str(where / "harness.cu"), str(where / "harness.so")
    with open(source, "w") as f:
        f.write(HARNESS)
    subprocess.run([build.NVCC] + build.ARCH + build.COMMON + [
        "--fmad=false", "-DLBIB_MEET_TRIES=20000u", "-I" + build.CSRC, "-shared", "-cudart", "static", source, "-o",
        library], check=True)
    L = ctypes.CDLL(library)
    function = L.meet
    function.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint, ctypes.c_void_p]
    L.grid.argtypes = [ctypes.c_int, ctypes.c_void_p]

    def call(compaction, beside, missing):
        out = (ctypes.c_int * 10)()
        assert function(compaction, beside, missing, out) == 0
        keys = ("err", "errStage", "halt", "haltStage", "changed", "removed", "ran_out", "ringStart", "err2",
                "changed2")
        return dict(zip(keys, out))

    def grid(blocks):
        most = ctypes.c_int()
        return L.grid(blocks, ctypes.byref(most)), most.value
    call.grid = grid
    return call


def test_all_arrive(meet):
    got = meet(0, 1, 0)
    assert (got["err"], got["halt"], got["changed"], got["ran_out"], got["ringStart"]) == (0, 0, 0, 0, 0)
    got = meet(1, 0, 0)
    assert (got["err"], got["halt"], got["changed"], got["removed"], got["ran_out"]) == (0, 0, 1, 0, 0)


@pytest.mark.parametrize("compaction, beside", [(0, 0), (0, 1), (1, 0)],
                         ids=["ring order", "ring order beside", "compaction"])
def test_a_wait_that_runs_out(meet, compaction, beside):
    got = meet(compaction, beside, 3)
    assert got["err"] == ERR_STATE
    stage = ST_COARSEN if compaction else ST_BIO
    if beside:
        assert (got["halt"], got["errStage"]) == (0, stage)
    else:
        assert (got["halt"], got["haltStage"]) == (1, stage)
    # left at the first meeting: nothing of the later phases is written
    assert (got["changed"], got["removed"], got["ringStart"]) == (1, 1, 5)
    assert got["ran_out"] == 1
    # the next launch leaves at once, without another error
    assert (got["err2"], got["changed2"]) == (0, 1)


def test_grid_fits_the_device(meet):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    e, most = meet.grid(0)
    assert e == 0 and sms <= most <= 2 * sms and most % sms == 0
    e, _ = meet.grid(most * 64)
    assert e == 720  # cudaErrorCooperativeLaunchTooLarge
    assert meet.grid(0)[0] == 0

"""CPU checks of what the tiled kernel's host and device sides share (csrc/esmm_tiled_layout.h), compiled with the host compiler, and of
source rules that no GPU run can show without faulting."""
import ctypes as C
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "esmm-research_b200", "csrc")

SHIM = r"""
#include "esmm_tiled_layout.h"
using namespace esmm;
extern "C" void layout(int stages, int stage_bytes, int cap, int blocks, unsigned *out)
{
    const PackedSmem L = packed_smem_layout(stages, stage_bytes, cap, blocks != 0);
    const unsigned v[] = {L.stage_off, L.krow_off, L.krow_stride, L.rmask_off, L.rmask_stride, L.wlist_off, L.bar_off, L.misc_off, L.total};
    for (int i = 0; i < 9; ++i) out[i] = v[i];
}
extern "C" int pays(int work, int slots, int sixteenths) { return block_mode_pays(work, slots, sixteenths); }
extern "C" int pipeline_pays(int work, int slots, int rows64, int listed, int span, int shape)
{
    return row_major_pipeline_pays(work, slots, rows64, listed, span, shape);
}
extern "C" int shape(int M, int N, long tiles, long pairs, int sms) { return row_major_shape(M, N, tiles, pairs, sms); }
extern "C" int tail(int mine) { return block_tail(mine); }
extern "C" int constant(int i)
{
    const int v[] = {SMEM_LIMIT, BM_SMEM, PSTAGE_BYTES, P_MAX_STAGES, P_CONSUMER_WARPS, RM_STAGE_A_BYTES + STAGE_HALF_BYTES};
    return v[i];
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    src, so = d / "shim.cpp", d / "shim.so"
    src.write_text(SHIM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CSRC, "-o", str(so), str(src)])
    return C.CDLL(str(so))


def test_shared_memory_layout(shim):
    """For every ring depth and K: the regions follow one another, 16-byte (barriers: 8-byte) aligned; in a kernel with block mode
    the barriers and what follows them lie past the rings that block mode lays over the rest, whose memory may not hold live
    mbarriers; and block mode refuses no K that the pipeline alone takes."""
    limit, bm_smem, packed_stage, max_stages, warps, rm_stage = (shim.constant(i) for i in range(6))
    out = (C.c_uint * 9)()
    for stage in (packed_stage, rm_stage):
        for stages in range(2, max_stages + 1):
            for cap in list(range(64, 2048, 32)) + list(range(2048, 30000, 416)) + [27520, 27552]:
                totals = {}
                for blocks in (0, 1):
                    shim.layout(stages, stage, cap, blocks, out)
                    st, krow, krow_stride, rmask, rmask_stride, wlist, bar, misc, total = out
                    assert st == 0 and stage % 128 == 0 and krow >= stages * stage and krow_stride >= 2 * cap
                    assert rmask >= krow + 2 * krow_stride and rmask_stride >= cap
                    assert wlist >= rmask + 2 * rmask_stride and wlist % 16 == 0
                    assert bar >= wlist + warps * 2 * 96 and bar % 8 == 0
                    assert misc >= bar + (2 * max_stages + 4) * 8 and misc % 4 == 0 and total >= misc + 7 * 4
                    if blocks:
                        assert bar >= bm_smem, (stages, cap)
                    totals[blocks] = total
                assert (totals[0] <= limit) == (totals[1] <= limit), (stages, cap)


def test_block_mode_rule(shim):
    """Block mode where at most so many sixteenths of the sampled slots are live; never on samples that hold no live k at all (the
    rest of the operands may be dense).  The largest counts, 8 samples of 1024 k and 16 blocks, stay inside 32 bits."""
    for sixteenths in (4, 11):
        assert not shim.pays(0, 0, sixteenths)
        assert shim.pays(0, 16, sixteenths)
        top = 8 * 1024 * 16
        for slots in (16, 160, top):
            assert shim.pays(slots * sixteenths // 16, slots, sixteenths)
            assert not shim.pays(slots * sixteenths // 16 + 1, slots, sixteenths)
            assert not shim.pays(slots, slots, sixteenths)


def test_items_cut_in_halves(shim):
    """Block mode's end: twelve warps that draw a CTA's items, pairs first, then single blocks at 0.55 of a pair, finish no later (0.15 of a pair)
    than with four or six of the last items cut in halves, whichever is better."""
    def finish(mine, tail):
        warps = [0.0] * 12
        for cost in [1.0] * (mine - tail) + [0.55] * (2 * tail):
            i = warps.index(min(warps))
            warps[i] += cost
        return max(warps)

    for mine in range(1, 300):
        tail = shim.tail(mine)
        assert 0 <= tail <= mine
        if mine > 12:
            assert finish(mine, tail) <= min(finish(mine, 4), finish(mine, 6)) + 0.15, mine


def test_row_major_rule(shim):
    """Row-major A: which problems stay with the pipeline although their share of live slots is one for block mode.  Samples as the kinds of operands
    give them (per k looked at: listed, work and rows64 of a tile of 4 x 4 blocks), shapes on 148 SMs, and the side each was measured on."""
    shim.shape.argtypes = [C.c_int, C.c_int, C.c_long, C.c_long, C.c_int]
    span = 8 * 1024

    def pipeline(M, N, rows, gran, pa, pb):
        across = -(-N // 128)
        tiles = -(-M // rows) * across
        ra, rb = -(-M // 32), -(-N // 32)
        pairs = max(-(-ra // 2) * rb, ra * -(-rb // 2))
        na, nb = (2, 2) if gran == 64 else (4, 4)                       # patterns of their own per tile
        listed = span * (1 - (1 - pa) ** na) * (1 - (1 - pb) ** nb)
        work = span * 16 * pa * pb
        rows64 = span * 8 * pb * (pa if gran == 64 else 1 - (1 - pa) ** 2)
        return bool(shim.pipeline_pays(int(work), int(16 * listed), int(rows64), int(listed), span, shim.shape(M, N, tiles, pairs, 148)))

    for shape in [(4096, 4096, 128), (2048, 2048, 128), (1024, 1024, 64), (512, 4096, 128), (2048, 11008, 128)]:
        assert pipeline(*shape, 64, 0.2, 0.2) and not pipeline(*shape, 64, 0.1, 0.1) and not pipeline(*shape, 64, 0.5, 0.5)
        assert not pipeline(*shape, 32, 0.5, 0.5) and not pipeline(*shape, 32, 0.2, 0.2)
        assert pipeline(*shape, 64, 0.3, 0.3) == (shape[0] == 1024)
    for shape, even in [((4096, 4096, 128), True), ((3000, 3000, 128), True), ((512, 4096, 128), True), ((2048, 2048, 128), False), ((2048, 11008, 128), False)]:
        assert pipeline(*shape, 32, 0.7, 0.7) == even and pipeline(*shape, 32, 1.0, 0.4) == even
    assert not pipeline(3000, 3000, 128, 64, 0.2, 0.2)                  # ragged, many pairs
    assert pipeline(1100, 700, 64, 64, 0.2, 0.2) and pipeline(1100, 700, 64, 64, 0.2, 0.6)      # ragged, single blocks all
    assert not pipeline(1000, 1508, 128, 64, 0.3, 0.3)                  # 96 tiles
    assert not any(pipeline(64, 4096, 64, 32, pa, pb) for pa, pb in [(0.7, 0.7), (1.0, 0.4)])   # 32 tiles
    assert not pipeline(128, 2048, 128, 64, 0.2, 0.2)


def test_copies_that_signal_a_barrier_are_waited_for():
    """Row-major producers' cp.async copies signal the stage's barrier and are never committed to a group, so waiting for committed
    groups does not wait for them; a producer that leaves after a wait that ran out must wait for all of its copies."""
    text = open(os.path.join(CSRC, "esmm_gemm_tiled.cuh")).read()
    assert "cp.async.mbarrier.arrive.noinc" in text and "cp_async_commit" not in text
    assert not re.search(r"cp_async_wait_group<", text)
    assert re.search(r"if \(RM\) cp_async_wait_all\(\);", text)

"""The prefill GEMM's choice of schedule and tile height (mlx_b200/csrc/qmm_plan.h), compiled for the host."""
import ctypes as C
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx_b200", "csrc")
SHIM = """
#include "qmm_plan.h"
extern "C" int plan(int M, int K, int N, int bits, int group, int y_bf16, int sharded, int ld, int col0, int sms, int streamk, int pair, int* out) {
    luxcuda::GemmPlan p{};
    if (!luxcuda::choose_gemm_plan({M, K, N, bits, group, y_bf16 != 0, sharded != 0, ld, col0}, sms, {streamk, pair}, false, &p)) return 0;
    const int v[] = {p.bm, p.m_tiles, p.n_tiles, p.streamk, p.pair, p.w_slots, p.y_tma, (int)p.smem};
    for (int i = 0; i < 8; i++) out[i] = v[i];
    return 1;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(d / "shim.cpp"), "-o", str(d / "plan.so")], check=True)
    f = C.CDLL(str(d / "plan.so")).plan

    def call(M, K, N, bits=4, group=64, y_bf16=True, shard=None, sms=148, streamk=-1, pair=-1):
        out = (C.c_int * 8)()
        ok = f(M, K, N, bits, group, int(y_bf16), int(shard is not None), *(shard or (N, 0)), sms, streamk, pair, out)
        return dict(zip(("bm", "m_tiles", "n_tiles", "streamk", "pair", "w_slots", "y_tma", "smem"), out)) if ok else None
    return call


def test_every_plan_can_be_launched(plan):
    """Heights that the matrix instructions are documented for (pairs of CTAs: multiples of 32; one CTA: of 16), tile rows
    that cover M and are none of them empty, shared memory within a CTA's 227 KB, a slot of weights per group."""
    rng = random.Random(3)
    pairs = 0
    for _ in range(4000):
        M, N = int(17 * 241 ** rng.random()), int(300 ** rng.random() * 100)
        bits, group = rng.choice([4, 8]), rng.choice([32, 64, 128])
        K = max(64, group) * rng.randint(1, 128)
        shard = rng.choice([None, None, (2 * N, N), (2 * N + 1, N)])
        for streamk, pair in ((-1, -1), (0, 0), (0, 1), (1, -1)):
            p = plan(M, K, N, bits, group, rng.random() < 0.7, shard, streamk=streamk, pair=pair)
            assert p is not None
            assert streamk < 0 or p["streamk"] == streamk
            assert streamk != 0 or p["pair"] == pair
            pairs += p["pair"]
            assert p["bm"] % (32 if p["pair"] else 16) == 0 and 16 <= p["bm"] <= 256, (M, K, N, p)
            assert (p["m_tiles"] - 1) * p["bm"] < M <= p["m_tiles"] * p["bm"]
            assert p["smem"] <= 227 * 1024 and 1 <= p["w_slots"] <= 4
    assert pairs > 4000  # (a quarter of the plans are forced to pairs)


def test_an_odd_number_of_sms_has_no_pairs(plan):
    assert plan(2048, 4096, 4096, sms=147, streamk=0, pair=1) is None
    assert plan(2048, 4096, 4096, sms=147)["pair"] == 0


@pytest.mark.parametrize("group", [32, 64, 128])
def test_many_rows_take_pairs_whatever_the_group(plan, group):
    """2048 x 2880 x 11008 and 2048 x 1024 x 4096 in groups of 32: 100 and 21 us by pairs, 108 and 23 by single CTAs."""
    for K, N in ((2880, 11008), (1024, 4096)):
        if K % group == 0:
            assert plan(2048, K, N, group=group)["pair"] == 1


def test_smoke_runs_each_of_the_three_kernels(plan):
    import __graft_entry__
    for name, (M, K, N) in __graft_entry__.SMOKE_PREFILL.items():
        p = plan(M, K, N)
        assert name == ("qmm_tc<4,stream-k>" if p["streamk"] else "qmm_tc<4,pairs>" if p["pair"] else "qmm_tc<4>")

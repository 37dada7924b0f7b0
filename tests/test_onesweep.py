"""The one-sweep decode kernel: its schedule on the CPU, its results against the oracle on a B200."""
import ctypes as C
import math
import os
import re
import subprocess

import pytest
import torch

from conftest import ROOT, assert_parity
from oracle import oracle_colreduce

HARNESS = r"""
#include "plan.h"
extern "C" int chunks_of(int B, int H, int M, int N, int D, int causal, int dtype, int sms, long long* out) {
  fcr_problem p{};
  p.B = B; p.H = H; p.M = M; p.N = N; p.D = D;
  const int64_t qs[4] = {(int64_t)H * M * D, (int64_t)M * D, D, 1}, ks[4] = {(int64_t)H * N * D, (int64_t)N * D, D, 1};
  for (int i = 0; i < 4; ++i) { p.q_strides[i] = qs[i]; p.k_strides[i] = ks[i]; }
  p.in_dtype = dtype; p.is_causal = causal; p.causal_offset = -1; p.scale = 1.f;
  fcr_plan pl;
  std::string err;
  if (fcr::plan_problem(p, sms, pl, err) != FCR_OK) return -1;
  out[0] = pl.key_stream; out[1] = pl.score_cache; out[2] = pl.d_pad; out[3] = pl.n_pad / 128; out[4] = pl.m_pad;
  out[5] = pl.workspace_bytes; out[6] = fcr::onesweep_bytes(p, pl, sms); out[7] = fcr::onesweep_counter_bytes(p);
  out[8] = pl.off_part_l + 4ll * pl.row_splits * B * H * pl.m_pad;
  return fcr::onesweep_chunks(p, pl, sms);
}
extern "C" void item_of(int S, int key_tiles, int item, int* out) {
  fcr::keystream_item(S, key_tiles, item, out[0], out[1], out[2], out[3]);
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("onesweep")
    (d / "harness.cpp").write_text(HARNESS)
    so = d / "harness.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "flash_colreduce_b200", "csrc"),
                    "-o", str(so), str(d / "harness.cpp")], check=True)
    lib = C.CDLL(str(so))

    def plan(b, h, m, n, d, causal=1, dtype=0, sms=148):
        out = (C.c_longlong * 9)()
        return lib.chunks_of(b, h, m, n, d, causal, dtype, sms, out), list(out)

    def item(s, tiles, i):
        out = (C.c_int * 4)()
        lib.item_of(s, tiles, i, out)
        return tuple(out)

    return plan, item


@pytest.mark.parametrize("b,h,m,n,sms", [(1, 1, 17, 1024, 148), (1, 1, 128, 90000, 148), (1, 1, 64, 70000, 3), (1, 3, 100, 9000, 7),
                                         (16, 32, 64, 16384, 148), (1, 32, 128, 4096, 148), (2, 75, 33, 1027, 148), (1, 2, 40, 2000, 1), (2, 75, 32, 6000, 148),
                                         (1, 40, 40, 13000, 100)])
def test_schedule_covers_the_keys_and_never_waits_in_a_circle(planner, b, h, m, n, sms):
    """Walks every CTA as the kernel does: its folding warps take rows segment n, then columns segment n - 1 (which
    needs the lse values of that chunk); a team of statistics warps publishes chunk n once it is folded, then fetches
    its lse values (which needs every chunk of the head published).  All must reach their end."""
    plan, item = planner
    S, info = plan(b, h, m, n, 128, sms=sms)
    tiles, bh = info[3], b * h
    assert 1 <= S <= min(tiles, sms)
    items, G = bh * S, min(bh * S, sms)
    seen = {}
    for i in range(items):
        head, sp, lo, hi = item(S, tiles, i)
        assert head == i // S and sp == i % S and lo < hi
        seen.setdefault(head, []).extend(range(lo, hi))
    assert all(seen[x] == list(range(tiles)) for x in range(bh))
    chunks = [(items - c + G - 1) // G for c in range(G)]
    copies, lag, buffers = (4 if m <= 32 else 2 if m <= 64 else 1), 1, 4
    fold, counted, published, fetched = [0] * G, [0] * bh, [set() for _ in range(G)], [set() for _ in range(G)]
    stat = [[0] * copies for _ in range(G)]  # steps done by each team: even ones publish a chunk, odd ones fetch
    moved = True
    while moved:
        moved = False
        for c in range(G):
            for team in range(copies):
                while team + copies * (stat[c][team] >> 1) < chunks[c]:
                    n = team + copies * (stat[c][team] >> 1)
                    head = (c + n * G) // S
                    if stat[c][team] & 1:
                        if counted[head] < S or (n >= buffers and fold[c] < 2 * (n - buffers + lag) + 2):
                            break
                        fetched[c].add(n)
                    else:
                        if fold[c] < 2 * n + 1:
                            break
                        published[c].add(n)
                        counted[head] += 1
                    stat[c][team] += 1
                    moved = True
            while fold[c] < 2 * (chunks[c] + lag):
                n = (fold[c] >> 1) - (fold[c] & 1) * lag
                if 0 <= n < chunks[c]:
                    if fold[c] & 1:
                        if n not in fetched[c]:
                            break
                    elif n >= buffers and n - buffers not in published[c]:
                        break
                fold[c] += 1
                moved = True
    assert all(fold[c] == 2 * (chunks[c] + lag) and len(fetched[c]) == chunks[c] for c in range(G)), "a CTA waits for good"


def test_the_exchange_orders_the_memory_of_all_lanes():
    """One lane of a statistics warp releases and acquires a head's counter for the loads and stores of all 32: a warp
    barrier stands between the stores of a chunk state and the release, and between the acquire and the loads."""
    with open(os.path.join(ROOT, "flash_colreduce_b200", "csrc", "onesweep_sm100.cuh")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert code.count("red_release_add(") == 1 and code.count("__stcg(") == 1 and code.count("__ldcg(") == 1
    publish = code[code.index("__stcg("):code.index("red_release_add(")]
    collect = code[code.rindex("ld_acquire("):code.index("__ldcg(")]
    assert "__syncwarp()" in publish and "__syncwarp()" in collect


def test_which_shapes_take_it_and_where_its_scratch_lies(planner):
    plan, _ = planner
    for m, n, d, dtype, takes in [(17, 1024, 128, 0, True), (128, 1024, 64, 0, True), (64, 4096, 80, 1, True), (64, 4096, 64, 2, True),
                                  (16, 4096, 128, 0, False),   # score cache
                                  (64, 4096, 129, 0, False), (64, 4096, 72, 2, False),  # rows beyond 256 bytes
                                  (64, 800000, 128, 0, False),  # too few, too long heads: a chunk would outgrow the L2
                                  (129, 4096, 128, 0, False), (64, 895, 128, 0, False)]:  # not key streaming
        S, info = plan(2, 3, m, n, d if dtype == 2 else (d + 7) // 8 * 8, dtype=dtype)
        assert (S > 0) == takes
        if takes:
            need = info[7] + (S * 6 * info[4] * 8 + 255) // 256 * 256
            assert info[6] == need and info[7] >= 6 * 4 * 4
            assert info[5] - info[6] >= info[8] and (info[5] - info[6]) % 256 == 0  # after the partial states
        else:
            assert info[6] == 0


def _call(nat, qd, kd, red, causal, scale, ws_bytes=None):
    b, h, m, d = qd.shape
    n = kd.shape[2]
    dt = {torch.float16: nat.FCR_F16, torch.bfloat16: nat.FCR_BF16, torch.float32: nat.FCR_F32}[qd.dtype]
    pr = nat.make_problem(b, h, m, n, d, qd.stride(), kd.stride(), dt, nat.REDUCTION_CODES[red], causal, scale)
    pl = nat.plan(pr, 0)
    ws = torch.empty(ws_bytes or pl.workspace_bytes, dtype=torch.uint8, device=qd.device)
    ws.fill_(0xAB)  # nothing in the workspace may be taken for granted
    out = torch.full((b, h, n), float("nan"), dtype=torch.float32, device=qd.device)
    before = nat.lib.fcr_launch_count()
    stream = torch.cuda.current_stream().cuda_stream
    nat.check(nat.lib.fcr_colreduce(C.byref(pr), qd.data_ptr(), kd.data_ptr(), out.data_ptr(), nat.FCR_F32, ws.data_ptr(),
                                    ws.numel(), stream), "fcr_colreduce")
    nat.check(nat.lib.fcr_read_device_status(ws.data_ptr(), stream, None), "device status")
    return out, nat.lib.fcr_launch_count() - before, pl, pr


@pytest.mark.gpu
@pytest.mark.parametrize("b,h,m,n,d,dtype", [(1, 1, 17, 1024, 128, "fp16"),   # least queries, least key tiles
                                             (2, 3, 32, 1025, 64, "bf16"),    # a whole lane group, one key past a tile
                                             (1, 5, 33, 3000, 80, "fp16"),    # one query in the second group
                                             (3, 50, 64, 1151, 128, "fp16"),  # several heads per CTA
                                             (2, 75, 32, 6000, 64, "bf16"),   # four teams, ten chunks per CTA
                                             (1, 2, 100, 20000, 64, "fp32"),  # TF32, long head
                                             (1, 160, 128, 1300, 128, "bf16"),
                                             (1, 1, 127, 70001, 128, "fp16")])  # one head over all CTAs, several chunks each
def test_one_sweep_matches_the_oracle_and_the_two_sweep_kernels(b, h, m, n, d, dtype):
    from flash_colreduce_b200 import _native as nat

    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(m * n)
    tt = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}[dtype]
    q = torch.randn(b, h, m, d, generator=g).to(torch.bfloat16 if dtype == "fp32" else tt).to(tt)  # exact in TF32
    k = torch.randn(b, h, n, d, generator=g).to(torch.bfloat16 if dtype == "fp32" else tt).to(tt)
    qd, kd = q.to(dev), k.to(dev)
    scale = -1.3 / math.sqrt(d) if m == 33 else 1 / math.sqrt(d)
    for red, causal in (("sum", True), ("mean", True), ("max", False), ("sum", False)):
        out, launches, pl, pr = _call(nat, qd, kd, red, causal, scale)
        assert launches == 1, "one kernel"
        assert_parity(out, oracle_colreduce(q, k, red, causal, scale=scale), red)
        again, _, _, _ = _call(nat, qd, kd, red, causal, scale)
        assert torch.equal(out, again)
        # the least workspace the call takes leaves no room for the chunk states: two sweeps, as accurate
        least = int(pl.off_part_l) + 4 * int(pl.row_splits) * b * h * int(pl.m_pad)
        two, launches, _, _ = _call(nat, qd, kd, red, causal, scale, ws_bytes=(least + 255) // 256 * 256)
        assert launches == 3
        # two fp32 evaluations of the same sums: each within 2^-18 of a column (lse of about 2^4 rounded to 2^-20,
        # two units of ex2, sums of at most 128 terms)
        torch.testing.assert_close(out, two, rtol=2.0 ** -17, atol=1e-9)


@pytest.mark.gpu
def test_one_sweep_under_graph_capture_and_on_two_streams():
    from flash_colreduce_b200 import flash_colreduce

    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(3)
    q = torch.randn(2, 40, 64, 128, generator=g, device=dev, dtype=torch.float16)
    k = torch.randn(2, 40, 5000, 128, generator=g, device=dev, dtype=torch.float16)
    old = os.environ.get("FCR_DEBUG_SYNC")
    os.environ["FCR_DEBUG_SYNC"] = "0"
    try:
        want = flash_colreduce(q, k, "sum", is_causal=True)
        s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        got = []
        for _ in range(20):  # cooperative launches of two streams wait for one another, never inside one another
            for s in (s1, s2):
                with torch.cuda.stream(s):
                    got.append(flash_colreduce(q, k, "sum", is_causal=True))
        torch.cuda.synchronize()
        assert all(torch.equal(x, want) for x in got)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = flash_colreduce(q, k, "sum", is_causal=True)
        out.zero_()
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    finally:
        if old is None:
            os.environ.pop("FCR_DEBUG_SYNC", None)
        else:
            os.environ["FCR_DEBUG_SYNC"] = old


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(64, 4096), (300, 700), (1100, 2100)])
@pytest.mark.parametrize("shape", ["rising", "falling", "spike", "flat", "tiny"])
def test_rows_whose_maximum_moves(m, n, shape):
    """Scores that rise or fall by hundreds along the keys, one key far above the rest, equal scores: the running
    maximum of a chunk, of a warpgroup and of a head each move by more than the exponent's range."""
    from flash_colreduce_b200 import _native as nat

    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(n)
    d = 64
    q = torch.randn(1, 2, m, d, generator=g).half()
    k = torch.randn(1, 2, n, d, generator=g).half() * 0.5
    q[..., 0] = 8.0
    ramp = torch.linspace(0.0, 60.0, n)
    k[..., 0] = {"rising": ramp, "falling": ramp.flip(0), "spike": torch.where(torch.arange(n) == n - 70, 60.0, 0.0),
                 "flat": torch.full((n,), 3.0), "tiny": torch.full((n,), -60.0)}[shape].half()
    for causal in (False, True):
        out, _, _, _ = _call(nat, q.to(dev), k.to(dev), "sum", causal, 1.0)
        want = oracle_colreduce(q, k, "sum", causal, scale=1.0)
        # fp32 scores of up to 500 carry 2^-15 absolute error into the exponent
        torch.testing.assert_close(out.cpu().double(), want.double(), rtol=2e-3, atol=1e-5)

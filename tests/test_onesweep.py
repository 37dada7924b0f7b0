"""The one-sweep decode kernel: its schedule on the CPU, its results against the oracle on a B200."""
import ctypes as C
import math
import os
import random
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
  out[5] = pl.workspace_bytes; out[6] = fcr::onesweep_bytes(p, pl, fcr::onesweep_chunks(p, pl, sms)); out[7] = fcr::onesweep_counter_bytes(p);
  out[8] = pl.off_part_l + 4ll * pl.row_splits * B * H * pl.m_pad;
  return fcr::onesweep_chunks(p, pl, sms);
}
extern "C" fcr::OneSweepDealer* dealer_new(int S, int n_items, int ticket) {
  auto* d = new fcr::OneSweepDealer;
  d->start(S, n_items, new int[fcr::kOneSweepHeld], ticket);
  return d;
}
extern "C" void dealer_free(fcr::OneSweepDealer* d) { delete[] d->held; delete d; }
extern "C" int dealer_finished(fcr::OneSweepDealer* d) { return d->finished(); }
extern "C" int dealer_needs_ticket(fcr::OneSweepDealer* d) { return d->needs_ticket(); }
extern "C" void dealer_draw(fcr::OneSweepDealer* d, int t) { d->draw(t); }
extern "C" int dealer_deal(fcr::OneSweepDealer* d, int* out) { d->deal(out[0], out[1]); return d->tail - d->head; }
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
    lib.dealer_new.restype = C.c_void_p
    for name in ("dealer_free", "dealer_finished", "dealer_needs_ticket", "dealer_draw", "dealer_deal"):
        getattr(lib, name).argtypes = [C.c_void_p] + {"dealer_draw": [C.c_int], "dealer_deal": [C.c_void_p]}.get(name, [])

    def plan(b, h, m, n, d, causal=1, dtype=0, sms=148):
        out = (C.c_longlong * 9)()
        return lib.chunks_of(b, h, m, n, d, causal, dtype, sms, out), list(out)

    def item(s, tiles, i):
        out = (C.c_int * 4)()
        lib.item_of(s, tiles, i, out)
        return tuple(out)

    return plan, item, lib


class _Cta:
    """One CTA of the kernel as agents that wait for one another: the TMA warp (deals records, fills the ring), the folding
    warps (with the MMA warps: a tile's slot is free once it is folded, which is later than in the kernel) and the teams of
    statistics warps.  Every agent is a generator that yields the condition it waits for."""

    def __init__(self, sim):
        self.sim, self.loaded, self.folded, self.records = sim, 0, 0, []
        self.folded_seg = [0, 0]             # rows and columns passes folded
        self.loaded_seg = [0, 0]
        self.parts_full, self.parts_read = 0, set()
        self.lse_full, self.lse_done = set(), 0
        self.agents = [self.tma(), self.fold()] + [self.stat(t) for t in range(sim.copies)]
        self.read = {x: -1 for x in range(1 + sim.copies)}  # the record at hand: of the folding warps, of each team

    def segment(self, item, kind):
        _, _, lo, hi = self.sim.item(self.sim.S, self.sim.tiles, item)
        yield lambda: self.folded_seg[kind] >= self.loaded_seg[kind]  # the query tile of this kind is free
        self.loaded_seg[kind] += 1
        for _ in range(lo, hi):
            yield lambda: self.loaded - self.folded < self.sim.ring
            self.loaded += 1

    def tma(self):
        sim, out = self.sim, (C.c_int * 2)()
        d = sim.lib.dealer_new(sim.S, sim.items, sim.draw())

        def announce():
            if sim.lib.dealer_finished(d):
                rec = None
            else:
                held = sim.lib.dealer_deal(d, out)
                assert held <= sim.S
                rec = (out[0], out[1])
                assert rec != (-1, -1)
            self.records.append(rec)
            return rec

        rec = announce()
        while rec is not None:
            need = sim.lib.dealer_needs_ticket(d)
            if rec[0] >= 0:
                yield from self.segment(rec[0], 0)
            if need:
                sim.lib.dealer_draw(d, sim.draw())
            yield lambda: len(self.records) - max(0, min(self.read.values())) < 16
            cols, rec = rec[1], announce()
            if cols >= 0:
                yield from self.segment(cols, 1)
        sim.lib.dealer_free(d)

    def next_record(self, reader):
        self.read[reader] += 1  # the one before is given back
        yield lambda: len(self.records) > self.read[reader]
        return self.records[self.read[reader]]

    def fold(self):
        n_rows = n_cols = 0
        while (rec := (yield from self.next_record(0))) is not None:
            for kind in (0, 1):
                if rec[kind] < 0:
                    continue
                head, _, lo, hi = self.sim.item(self.sim.S, self.sim.tiles, rec[kind])
                if kind == 1:
                    yield lambda: n_cols in self.lse_full
                    assert self.sim.counted[head] == self.sim.S
                for _ in range(lo, hi):
                    yield lambda: self.loaded > self.folded
                    self.folded += 1
                self.folded_seg[kind] += 1
                self.sim.swept[kind].append(rec[kind])
                if kind == 0:
                    yield lambda: n_rows < 4 or n_rows - 4 in self.parts_read
                    n_rows += 1
                    self.parts_full = n_rows
                else:
                    n_cols += 1
                    self.lse_done = n_cols

    def stat(self, team):
        sim, n_rows, n_cols = self.sim, 0, 0
        while (rec := (yield from self.next_record(1 + team))) is not None:
            if rec[1] >= 0:
                if n_cols % sim.copies == team:
                    head = rec[1] // sim.S
                    yield lambda: sim.counted[head] == sim.S
                    yield lambda: n_cols < 4 or self.lse_done > n_cols - 4
                    self.lse_full.add(n_cols)
                n_cols += 1
            if rec[0] >= 0:
                if n_rows % sim.copies == team:
                    yield lambda: self.parts_full > n_rows
                    self.parts_read.add(n_rows)
                    sim.counted[rec[0] // sim.S] += 1
                n_rows += 1


class _Sim:
    def __init__(self, lib, item, S, tiles, heads, m, ring, seed):
        self.lib, self.item, self.S, self.tiles, self.items, self.ring = lib, item, S, tiles, heads * S, ring
        self.copies = 4 if m <= 32 else 2 if m <= 64 else 1
        self.counted, self.swept, self.tickets = [0] * heads, ([], []), 0
        self.rng = random.Random(seed)

    def draw(self):
        self.tickets += 1
        return self.tickets - 1

    def run(self, grid, room):
        """`grid` CTAs, of which `room` run at a time: the next one starts when one has ended."""
        live, started = [], 0
        while started < grid or live:
            while started < grid and len(live) < room:
                live.append([[g, None] for g in _Cta(self).agents])
                started += 1
            moved = False
            self.rng.shuffle(live)
            for cta in live:
                for agent in list(cta):
                    steps = 0
                    while agent[1] is None or agent[1]():
                        moved, steps = True, steps + 1
                        try:
                            agent[1] = next(agent[0])
                        except StopIteration:
                            cta.remove(agent)
                            break
                        if steps > self.rng.randrange(1, 40):
                            break
            if any(not cta for cta in live):
                live = [cta for cta in live if cta]
                moved = True
            assert moved, "CTAs wait for good"


@pytest.mark.parametrize("b,h,m,n,sms,room", [(1, 1, 17, 1024, 148, 148), (1, 1, 128, 90000, 148, 148), (1, 1, 128, 90000, 148, 1),
                                              (1, 1, 64, 70000, 3, 3), (1, 3, 100, 9000, 7, 7), (1, 3, 100, 9000, 7, 2),
                                              (4, 32, 64, 16384, 148, 148), (1, 32, 64, 16384, 148, 147), (1, 32, 64, 16384, 148, 1),
                                              (1, 32, 128, 4096, 148, 148), (1, 32, 128, 4096, 148, 100), (1, 32, 128, 4096, 148, 1),
                                              (2, 75, 33, 1027, 148, 148), (1, 2, 40, 2000, 1, 1), (2, 75, 32, 6000, 148, 148),
                                              (2, 75, 32, 6000, 148, 5), (1, 40, 40, 13000, 100, 100), (1, 8, 64, 32768, 148, 3)])
def test_every_chunk_is_swept_twice_however_few_ctas_run(planner, b, h, m, n, sms, room):
    """A call finishes on the SMs that are free: with room for one CTA, for some or for all of the grid, whoever draws the
    tickets first, no CTA waits for one that has not started, and each chunk has its rows and its columns pass once."""
    plan, item, lib = planner
    S, info = plan(b, h, m, n, 128, sms=sms)
    tiles, heads = info[3], b * h
    assert 1 <= S <= min(tiles, sms)
    seen = {}
    for i in range(heads * S):
        head, sp, lo, hi = item(S, tiles, i)
        assert head == i // S and sp == i % S and lo < hi
        seen.setdefault(head, []).extend(range(lo, hi))
    assert all(seen[x] == list(range(tiles)) for x in range(heads))
    sim = _Sim(lib, item, S, tiles, heads, m, ring=4, seed=n)
    sim.run(min(heads * S, sms), room)
    assert sorted(sim.swept[0]) == sorted(sim.swept[1]) == list(range(heads * S))


def test_the_exchange_orders_the_memory_of_all_lanes():
    """One lane of a statistics warp releases and acquires a head's counter for the loads and stores of all 32: a warp
    barrier stands between the stores of a chunk state and the release, and between the acquire and the loads."""
    with open(os.path.join(ROOT, "flash_colreduce_b200", "csrc", "onesweep_sm100.cuh")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert code.count("red_release_add(") == 1 and code.count("__stcg(") == 1 and code.count("__ldcg(") == 1
    publish = code[code.index("__stcg("):code.index("red_release_add(")]
    collect = code[code.rindex("ld_acquire("):code.index("__ldcg(")]
    assert "__syncwarp()" in publish and "__syncwarp()" in collect


def test_the_chunks_are_chosen_with_the_plan():
    """A repeated problem plans nothing: the search for the chunk count runs where a plan is made, not in every call."""
    with open(os.path.join(ROOT, "flash_colreduce_b200", "csrc", "colreduce_sm100.cu")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    planner, rest = code.split("static int plan_for_call(", 1)[1].split("\n}\n", 1)
    assert planner.count("onesweep_chunks(") == 1 and code.count("onesweep_chunks(") == 1


def test_which_shapes_take_it_and_where_its_scratch_lies(planner):
    plan, _, _ = planner
    for m, n, d, dtype, takes in [(17, 1024, 128, 0, True), (100, 90000, 64, 0, True), (128, 1024, 64, 0, True), (64, 4096, 80, 1, True), (64, 4096, 64, 2, True),
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
                                             (4, 80, 100, 2100, 64, "bf16"),  # short rows, K beyond the L2
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
        for _ in range(20):  # blocks of the one call start as blocks of the other end
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
def test_one_sweep_finishes_while_another_kernel_holds_an_sm():
    """A kernel of another stream (one block that waits for a load left out on purpose until its bound of about 0.2 s runs
    out) holds an SM that the call's grid would fill: the call ends on the others, with the same result."""
    from flash_colreduce_b200 import _native as nat

    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(9)
    q = torch.randn(1, 32, 128, 128, generator=g, device=dev, dtype=torch.float16)
    k = torch.randn(1, 32, 4096, 128, generator=g, device=dev, dtype=torch.float16)
    x = torch.randn(1, 1, 128, 64, generator=g, device=dev, dtype=torch.float16)
    out, launches, _, pr = _call(nat, q, k, "sum", True, 0.09)
    assert launches == 1
    one = nat.make_problem(1, 1, 128, 128, 64, x.stride(), x.stride(), nat.FCR_F16, nat.FCR_SUM, False, 0.125)
    pl = nat.plan(one, 0)
    assert pl.row_ctas == 1
    ws = torch.empty(int(pl.workspace_bytes), dtype=torch.uint8, device=dev)
    small = torch.empty(1, 1, 128, dtype=torch.float32, device=dev)
    holder, other, held = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    nat.check(nat.lib.fcr_self_test_hooks(400_000_000, 0), "fcr_self_test_hooks")
    try:
        nat.check(nat.lib.fcr_colreduce(C.byref(one), x.data_ptr(), x.data_ptr(), small.data_ptr(), nat.FCR_F32, ws.data_ptr(),
                                        ws.numel(), holder.cuda_stream), "fcr_colreduce")
    finally:
        nat.check(nat.lib.fcr_self_test_hooks(0, -1), "fcr_self_test_hooks")
    held.record(holder)
    with torch.cuda.stream(other):
        got, _, _, _ = _call(nat, q, k, "sum", True, 0.09)  # waits for its own stream
        still_held = not held.query()
    torch.cuda.synchronize()
    code = C.c_int32(0)
    assert nat.lib.fcr_poll_device_status(C.byref(code)) == nat.FCR_ERR_DEVICE_TIMEOUT  # the holder's report
    assert still_held, "the call waited for the other kernel's SM"
    assert torch.equal(got, out)


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

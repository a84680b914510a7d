"""What a context keeps between calls: tables of an index since rebuilt, buffers
under a tight budget, calls that failed half way (B200 only).
"""
import threading
from ctypes import byref, c_void_p

import numpy as np
import pytest

from swiftimpute_b200 import _native as N
from swiftimpute_b200 import synth
from swiftimpute_b200.engine import Engine

pytestmark = pytest.mark.gpu

ERR_STATE, ERR_BUDGET = 5, 7


def noalloc(torch, eng, codes, p):
    """si_impute_device_noalloc: its status and the dosage it wrote."""
    g = torch.from_numpy(codes).cuda()
    dos = torch.zeros(codes.shape, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    st = eng.lib.si_impute_device_noalloc(eng.h, byref(p), c_void_p(g.data_ptr()), codes.shape[0],
                                          c_void_p(dos.data_ptr()), None, None, None)
    torch.cuda.synchronize()
    return st, dos.cpu().numpy()


def small(seed=1, M=600, N_=300, B=16):
    panel, pos, _ = synth.make_panel(M, N_, 12, seed=seed, spacing=100)
    codes, _, _ = synth.make_targets(panel, B, synth.typed_every(M, 5), seed=seed + 1)
    return panel, pos, codes


@pytest.mark.parametrize("kind", [N.SEL_AUTO, N.SEL_FIRST_PAIRS])
def test_noalloc_after_a_rebuild(kind):
    """Tables of an index since rebuilt, or whose rebuild failed, are not set-up: the call is refused until an
    allocating call has filled them."""
    torch = pytest.importorskip("torch")
    panel, pos, codes = small()
    M, N_ = panel.shape
    p = N.default_params(num_states=8, ne=10000, selection_kind=kind)
    with Engine(0) as eng:
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        eng.impute(codes, p)
        st, first = noalloc(torch, eng, codes, p)
        assert st == N.SI_OK
        eng.pbwt_build()
        assert noalloc(torch, eng, codes, p)[0] == ERR_STATE
        eng.impute(codes, p)
        st, again = noalloc(torch, eng, codes, p)
        assert st == N.SI_OK and np.array_equal(first, again)
        used = eng.memory()[0]
    with Engine(0, hbm_budget_bytes=used + M * N_ * 2) as eng:  # no room for prefix rows
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        eng.impute(codes, p)
        assert noalloc(torch, eng, codes, p)[0] == N.SI_OK
        with pytest.raises(N.SIError):
            eng.pbwt_build(store_index=True)
        assert noalloc(torch, eng, codes, p)[0] == ERR_STATE


@pytest.mark.parametrize("room", ["pairs", "masks", "weights"])
def test_selection_that_does_not_fit(room):
    """A selection whose tables run out of budget half way is refused every time it is asked for, after a rebuild
    of the index too, holds nothing, and is right once there is room."""
    L = 16
    panel, pos, codes = small(seed=3, M=3000, N_=100, B=4)
    if room == "weights":  # the last table: allele bytes of a panel with others than 0 and 1
        panel = panel.copy()
        panel[::7, ::5] = 255
    M = panel.shape[0]

    def up(nbytes):
        return -(-nbytes // 256) * 256

    parts = [up(M * L * 8), up(M * 16), up(M * L * 8)]  # pairs, masks, weights
    with Engine(0) as eng:
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        base = eng.memory()[0]
        want = eng.select_states(L)
        whole = eng.memory()[0] - base
    have = sum(parts[:["pairs", "masks", "weights"].index(room) + 1])
    assert have < whole
    with Engine(0, hbm_budget_bytes=base + have + 256) as eng:
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        for rebuild in (False, False, True, False):
            if rebuild:
                eng.pbwt_build()
            with pytest.raises(N.SIError) as e:
                eng.select_states(L)
            assert e.value.status == ERR_BUDGET
            assert eng.memory()[0] == base
        assert np.array_equal(eng.select_states(1)[:, 0], want[:, 0])  # what fits beside it is served
    with Engine(0, hbm_budget_bytes=base + whole) as eng:
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        for _ in range(2):
            assert np.array_equal(eng.select_states(L), want)
            eng.pbwt_build()


def run_threads(works):
    """Each callable 1,000 times in a thread of its own; the first exception is raised here."""
    failed = []

    def loop(work):
        try:
            for _ in range(1000):
                work()
        except Exception as x:
            failed.append(x)

    threads = [threading.Thread(target=loop, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if failed:
        raise failed[0]


def test_imputations_in_two_threads():
    """A context each in two threads of a device, their kernels launched with different amounts of shared memory
    (outputs, checkpoint sizes): every call succeeds and is the same as alone."""
    panel, pos, codes = small(seed=5, M=60, N_=64, B=2)

    def params(C, flags=0):
        return N.default_params(num_states=8, ne=20000, flags=flags, checkpoint_interval=C, block_threads=128)

    chain = N.IMPUTE_FULL_CHAIN
    calls = [[(params(32, chain), True), (params(32, chain), False), (params(12), False)],
             [(params(8, chain), True), (params(8, chain), False), (params(2), False)]]
    with Engine(0) as one, Engine(0) as other:
        works = []
        for e, mine in zip((one, other), calls):
            e.upload_panel(panel); e.set_map(pos); e.pbwt_build()
            alone = [e.impute(codes, p, hap_prob=hp) for p, hp in mine]

            def work(e=e, mine=mine, alone=alone):
                for (p, hp), want in zip(mine, alone):
                    got = e.impute(codes, p, hap_prob=hp)
                    assert all(np.array_equal(got[k], want[k]) for k in want)

            works.append(work)
        run_threads(works)


def test_index_builds_in_two_threads():
    with Engine(0) as one, Engine(0) as other:
        works = []
        for e, N_ in ((one, 400), (other, 6000)):
            panel, _, _ = synth.make_panel(130, N_, 8, seed=N_)
            e.upload_panel(panel); e.pbwt_build()
            alone = e.select_states(8)

            def work(e=e, alone=alone):
                e.pbwt_build()
                assert np.array_equal(e.select_states(8), alone)

            works.append(work)
        run_threads(works)


def ends_bytes(B, M, lmax, C):
    """The full chain's ends at segments of C markers: alpha's, a 256-byte boundary, beta's and their units."""
    n = max(-(-M // C) - 1, 1)
    return -(-n * lmax * B * 4 // 256) * 256 + n * (lmax * 4 + 8) * B


def test_full_chain_makes_room_for_its_ends():
    """Under a budget whose room is held by tables of an index since rebuilt, the full chain's segments still run
    in parallel: the tables make room, and no one-pass checkpoints (which would count as used) are allocated."""
    panel, pos, codes = small(seed=7, M=1000, N_=64, B=500)
    chain = N.default_params(num_states=8, ne=20000, flags=N.IMPUTE_FULL_CHAIN)

    def before(eng):
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        eng.impute(codes, N.default_params(num_states=8, ne=20000))
        for L in range(9, 33):
            eng.select_states(L)
        full = eng.memory()[0]
        eng.pbwt_build()
        return full

    with Engine(0) as wide:
        full = before(wide)
        assert full - wide.memory()[0] > ends_bytes(500, 1000, 8, 16)  # the tables that wait
        want = wide.impute(codes, chain)
        used = wide.memory()[0]
    with Engine(0, hbm_budget_bytes=full + (64 << 10)) as tight:
        before(tight)
        got = tight.impute(codes, chain)
        assert tight.memory()[0] == used
    for key in want:
        assert np.array_equal(got[key], want[key])


def device_call(torch, eng, codes, p):
    """A full-chain call on device buffers of a stream of its own, warmed up: (stream, dosage, the call)."""
    g = torch.from_numpy(codes).cuda()
    dos = torch.zeros(codes.shape, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def call():
        eng.impute_device(g.data_ptr(), codes.shape[0], p, dos.data_ptr(), None, None, stream=stream.cuda_stream)

    call()
    torch.cuda.synchronize()
    return stream, dos, call


def capture(torch, stream, call):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        call()
    torch.cuda.synchronize()
    return graph


def test_full_chain_keeps_ends_that_fit():
    """Under a budget for the ends of whole default segments but not of half ones, a repeated call neither frees
    nor allocates: it can be captured."""
    torch = pytest.importorskip("torch")
    panel, pos, codes = small(seed=8, M=1000, N_=64, B=500)
    p = N.default_params(num_states=8, ne=20000, flags=N.IMPUTE_FULL_CHAIN | N.IMPUTE_RESELECT)
    whole, half = ends_bytes(500, 1000, 8, 32), ends_bytes(500, 1000, 8, 16)
    with Engine(0) as wide:
        wide.upload_panel(panel); wide.set_map(pos); wide.pbwt_build()
        _, want, _ = device_call(torch, wide, codes, p)
        used = wide.memory()[0]
    with Engine(0, hbm_budget_bytes=used + (whole + half) // 2) as tight:
        tight.upload_panel(panel); tight.set_map(pos); tight.pbwt_build()
        stream, dos, call = device_call(torch, tight, codes, p)
        assert torch.equal(dos, want) and tight.memory()[0] == used  # in parallel
        graph = capture(torch, stream, call)
        dos.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(dos, want)
        del graph


def test_captured_full_chain_keeps_its_ends():
    """The ends whose address a captured call holds are no room for other allocations: the graph replays right
    after the budget has been filled with tables."""
    torch = pytest.importorskip("torch")
    panel, pos, codes = small(seed=9, M=1000, N_=64, B=500)
    p = N.default_params(num_states=8, ne=20000, flags=N.IMPUTE_FULL_CHAIN | N.IMPUTE_RESELECT)
    ends = ends_bytes(500, 1000, 8, 16)
    with Engine(0) as wide:
        wide.upload_panel(panel); wide.set_map(pos); wide.pbwt_build()
        _, want, _ = device_call(torch, wide, codes, p)
        used = wide.memory()[0]
    with Engine(0, hbm_budget_bytes=used + ends + (1 << 20)) as tight:
        tight.upload_panel(panel); tight.set_map(pos); tight.pbwt_build()
        stream, dos, call = device_call(torch, tight, codes, p)
        graph = capture(torch, stream, call)
        assert tight.memory()[0] >= used + ends  # no longer what another allocation can have
        for L in range(9, 33):
            try:
                tight.select_states(L)
            except N.SIError as e:
                assert e.status == ERR_BUDGET
        dos.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(dos, want)
        del graph


def test_index_build_within_its_budget_after_another_panel():
    """An index whose build just fits the budget is built after another panel's too, whose larger kept buffer
    makes room."""
    M, N_ = 640, 25_000  # 10 segments, swept by groups
    small_panel, _, _ = synth.make_panel(9600, 1500, 8, seed=10)  # 148 segments, sorted: 1.8 MB of orders
    rng = np.random.default_rng(11)
    words = rng.integers(0, 1 << 32, (M, -(-N_ // 32)), dtype=np.uint32) & rng.integers(0, 1 << 32, (M, -(-N_ // 32)), dtype=np.uint32)

    def build(eng):
        eng.upload_packed(words, N_)
        eng.pbwt_build(store_index=True)
        return eng.prefix_rows(M - 1, 1)

    with Engine(0) as wide:
        want = build(wide)
        used = wide.memory()[0]
    # groups' scratch and ranks of nine segments, the sort buffer, ten start orders and the jobs
    budget = used + 4 * N_ * (4 * 9 + 9 + 4 + 10) + 8192
    for first in (False, True):
        with Engine(0, hbm_budget_bytes=budget) as eng:
            if first:
                eng.upload_panel(small_panel); eng.pbwt_build()
            assert np.array_equal(build(eng), want)


@pytest.mark.parametrize("L,C", [(3, 0), (4, 0), (5, 0), (8, 0), (8, 7), (12, 0), (16, 0), (16, 32), (27, 0), (32, 0), (32, 8)])
@pytest.mark.parametrize("mode", ["first_gap", "per_gap", "target"])
def test_full_chain_one_pass(L, C, mode):
    """The one-pass kernel, which a budget without room for both directions' ends falls back to, and the parallel
    segments: the same bits. Which of them ran shows in the memory used, where only the one pass' own checkpoints
    count."""
    M, B = 1029, 301
    panel, pos, _ = synth.make_panel(M, 64, 8, seed=L + C, spacing=1000)
    rng = np.random.default_rng(L + C)
    pos = np.cumsum(rng.integers(1, 5000, M)).astype(np.uint64)
    codes = rng.integers(0, 8, (B, M)).astype(np.uint8)  # five cells of eight untyped
    p = N.default_params(num_states=L, ne=20000, flags=N.IMPUTE_FULL_CHAIN, checkpoint_interval=C,
                         transition_mode=N.TRANS_PER_GAP if mode == "per_gap" else N.TRANS_MATRIX0,
                         selection_kind=N.SEL_TARGET if mode == "target" else N.SEL_AUTO)

    def run(eng):
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build(store_index=True)
        return eng.impute(codes, p, hap_prob=True)

    lmax = next(x for x in (4, 8, 16, 32) if L <= x)
    c = C or (16 if lmax == 32 else 32)
    one = -(-(-(-M // c) - 1) * lmax * B * 4 // 256) * 256
    assert ends_bytes(B, M, lmax, c) > one + (64 << 10)
    with Engine(0) as wide:
        want = run(wide)
        used = wide.memory()[0]
    with Engine(0, hbm_budget_bytes=used + one + (64 << 10)) as tight:
        got = run(tight)
        assert tight.memory()[0] == used + one
    for key in want:
        assert np.array_equal(got[key], want[key]), key

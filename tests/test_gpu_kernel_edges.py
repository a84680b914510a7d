"""Kernels at the sizes where their tiles, blocks and rules of dispatch change
sides, against the CPU oracle (B200 only).

Bars as in the parity tests: dosage and P(hap=1) within 1e-4 of the FP64
oracle; argmax alleles equal wherever the oracle's choice is not within 1e-5 of
the tie threshold.
"""
import numpy as np
import pytest

import oracle
from swiftimpute_b200 import _native as N
from swiftimpute_b200 import synth

pytestmark = pytest.mark.gpu

TOL = 1e-4


def own_sites(codes_all, counts, seed):
    """Each target keeps the genotypes of its own random markers, counts[b] of them."""
    rng = np.random.default_rng(seed)
    codes = np.full_like(codes_all, 3)
    for b, n in enumerate(counts):
        at = rng.choice(codes_all.shape[1], size=n, replace=False)
        codes[b, at] = codes_all[b, at]
    return codes


def check(engine, panel, pos, codes, L, ne=20000, per_gap=False, **kw):
    engine.upload_panel(panel)
    engine.set_map(pos)
    engine.pbwt_build()
    p = N.default_params(num_states=L, ne=ne, transition_mode=N.TRANS_PER_GAP if per_gap else N.TRANS_MATRIX0, **kw)
    got = engine.impute(codes, p, hap_prob=True)
    pairs = engine.select_states(L)
    want = oracle.fb_batch(codes, pairs, panel, pos, L, ne, per_gap=per_gap, tie_eps=p.tie_eps)
    assert np.abs(got["dosage"] - want["dosage"]).max() <= TOL
    assert np.abs(got["hap_prob"] - want["hap_prob"]).max() <= TOL
    diff = (got["haps"] != want["haps_argmax"]).any(axis=1)
    if diff.any():
        flips = [oracle.fb_batch(codes, pairs, panel, pos, L, ne, per_gap=per_gap, tie_eps=p.tie_eps + d)["haps_argmax"]
                 for d in (-1e-5, 1e-5)]
        assert not (diff & ~(flips[0] != flips[1]).any(axis=1)).any()
    return got


# typed markers of the targets of a group: none, one, around the chain's block of
# eight (and four) anchors, and all; groups whose chains end at different anchors
@pytest.mark.parametrize("L,spacing", [(3, 1000), (8, 500_000), (8, 1000), (16, 1000), (32, 1000)])
def test_chain_blocks(engine, L, spacing):
    M = 300
    panel, pos, _ = synth.make_panel(M, 512, 20, seed=L, spacing=spacing)
    counts = [0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 299, 300, 64, 0, 8, 100,
              40, 41, 42, 43, 44, 300, 1, 2]  # a full group and a partial one
    codes_all, _, _ = synth.make_targets(panel, len(counts), np.arange(M), seed=L + 1)
    codes = own_sites(codes_all, counts, seed=L + 2)
    got = check(engine, panel, pos, codes, L)
    # a target alone, and all targets of one group equal: the same chain whatever runs beside it
    p = N.default_params(num_states=L, ne=20000)
    for b in (0, 8, 22):
        alone = engine.impute(codes[b:b + 1], p, hap_prob=True)
        same = engine.impute(np.repeat(codes[b:b + 1], 33, axis=0), p, hap_prob=True)
        for key in ("dosage", "hap_prob", "haps"):
            assert np.array_equal(alone[key][0], got[key][b])
            assert np.array_equal(same[key], np.repeat(got[key][b:b + 1], 33, axis=0))


# rows that start anywhere, lengths around the lists' chunks (16, 512) and segments (4,096), batches
# around a group, typed and untyped first and last markers, rows without any typed marker
@pytest.mark.parametrize("M", [1, 2, 15, 16, 17, 31, 33, 497, 511, 513, 1023, 4095, 4096, 4097, 4111, 4112, 8191, 8209])
def test_list_rows(engine, M):
    B = 33 if M < 1000 else 5
    panel, pos, _ = synth.make_panel(M, 256, 20, seed=M, spacing=500_000)
    codes_all, _, _ = synth.make_targets(panel, B, np.arange(M), seed=M + 1, het_range=(0.0, 1.0))
    rng = np.random.default_rng(M + 2)
    codes = own_sites(codes_all, rng.integers(0, min(M, 600) + 1, B), seed=M + 3)
    codes[0] = 3
    codes[1] = codes_all[1]
    codes[2, -1] = codes_all[2, -1]
    codes[3] = np.where(codes[3] == 3, rng.integers(3, 256, M), codes[3])  # any byte above 2 is a missing call
    check(engine, panel, pos, codes, 8)


# targets of one array (the lanes of a CTA in step, slot data staged) against the same targets beside
# others with sites of their own (each lane by itself): bit for bit the same, and the oracle's. Runs shorter
# and longer than the staged head of the tables (64), one past the tables (4,096), odd rows, partial groups.
@pytest.mark.parametrize("L,M,every,B,spacing", [(8, 333, 7, 33, 1000), (4, 1024, 64, 129, 1000), (3, 1000, 65, 31, 500_000),
                                                 (16, 700, 63, 64, 1000), (32, 515, 130, 40, 1000),
                                                 (8, 9001, 4500, 5, 1000), (8, 640, 1, 32, 500_000)])
@pytest.mark.parametrize("other_alleles", [False, True])
def test_posterior_walks(engine, L, M, every, B, spacing, other_alleles):
    panel, pos, _ = synth.make_panel(M, 384, 20, seed=M + L, spacing=spacing)
    codes, _, _ = synth.make_targets(panel, B, synth.typed_every(M, every), seed=M + 1, het_range=(0.0, 1.0))
    if other_alleles:
        u = np.random.default_rng(M).random(panel.shape)
        panel = panel.copy()
        panel[u < 0.02] = 255
        panel[(u >= 0.02) & (u < 0.03)] = 2
    check(engine, panel, pos, codes, L)
    all_codes, _, _ = synth.make_targets((panel != 0).astype(np.uint8), B, np.arange(M), seed=M + 2, het_range=(0.0, 1.0))
    mixed = np.empty((2 * B, M), np.uint8)
    mixed[0::2] = codes
    mixed[1::2] = own_sites(all_codes, np.random.default_rng(M).integers(0, M // 2, B), seed=M + 3)
    for kw in ({}, {"sampling": N.SAMPLE_PHILOX}):
        for out in ({"hap_prob": True}, {}, {"dosage": False}):
            p = N.default_params(num_states=L, ne=20000, **kw)
            alone = engine.impute(codes, p, **out)
            beside = engine.impute(mixed, p, **out)
            for key in alone:
                if key != "haps" or not kw:  # a draw is keyed by the row's sample id
                    assert np.array_equal(alone[key], beside[key][0::2]), (key, kw, out)


# runs longer than the run tables (4,096 markers) in the walk in step, two cells a step by the closed form: the
# oracle's, and bit for bit the lanes' own walk's
@pytest.mark.parametrize("L,M,every,B", [(4, 4099, 4099, 1), (3, 8400, 4097, 33), (8, 13001, 4333, 5), (16, 9000, 4500, 32),
                                         (32, 8777, 4388, 7)])
@pytest.mark.parametrize("spacing", [1000, 500_000])
def test_long_runs_in_step(engine, L, M, every, B, spacing):
    panel, pos, _ = synth.make_panel(M, 64, 8, seed=M + L, spacing=spacing)
    codes, _, _ = synth.make_targets(panel, B, synth.typed_every(M, every), seed=M + 1, het_range=(0.0, 1.0))
    check(engine, panel, pos, codes, L)
    mixed = np.repeat(codes, 2, axis=0)  # an extra site in every other row: the lanes of a warp are not in step
    mixed[1::2, M // 3] = 1
    for kw in ({}, {"sampling": N.SAMPLE_PHILOX}):
        for out in ({"hap_prob": True}, {}, {"dosage": False}):
            p = N.default_params(num_states=L, ne=20000, **kw)
            alone, beside = engine.impute(codes, p, **out), engine.impute(mixed, p, **out)
            for key in alone:
                if key != "haps" or not kw:  # a draw is keyed by the row's sample id
                    assert np.array_equal(alone[key], beside[key][0::2]), (key, kw, out)


def test_long_runs_in_step_time(engine):
    M, B = 9100, 32
    panel, pos, _ = synth.make_panel(M, 64, 8, seed=1, spacing=1000)
    engine.upload_panel(panel)
    engine.set_map(pos)
    engine.pbwt_build()
    p = N.default_params(num_states=8, ne=20000)

    def posterior_ms(every):
        codes, _, _ = synth.make_targets(panel, B, synth.typed_every(M, every), seed=2)
        return min((engine.impute(codes, p), engine.last_kernel_ms()[3])[1] for _ in range(5))

    # the same markers in runs past the tables and within them: 3.24 and 1.69 ms (5.83 with a cell a step)
    assert posterior_ms(4500) <= 2.6 * posterior_ms(4000)


# the full chain in parallel segments against the oracle and against one pass over the chain (the
# kernel that a budget without room for the segments' ends falls back to):
# lengths around the checkpoint segments, the staged blocks (8, 4) and code chunks (32), B around a warp
@pytest.mark.parametrize("L,M,B,C", [(8, 1, 3, 0), (8, 2, 33, 0), (8, 31, 5, 0), (8, 32, 31, 0), (8, 33, 32, 0),
                                     (3, 65, 7, 0), (8, 500, 40, 7), (16, 257, 33, 0), (32, 131, 35, 0),
                                     (32, 64, 3, 16), (4, 1000, 64, 1), (8, 1029, 130, 32)])
@pytest.mark.parametrize("per_gap", [False, True])
def test_full_chain_segments(engine, L, M, B, C, per_gap):
    panel, pos, _ = synth.make_panel(M, 256, 20, seed=M + L, spacing=1000)
    rng = np.random.default_rng(M)
    pos = np.cumsum(rng.integers(1, 5000, M)).astype(np.uint64)
    codes_all, _, _ = synth.make_targets(panel, B, np.arange(M), seed=M + 1, het_range=(0.0, 1.0))
    codes = own_sites(codes_all, rng.integers(0, M + 1, B), seed=M + 2)
    kw = {"flags": N.IMPUTE_FULL_CHAIN, "checkpoint_interval": C}
    got = check(engine, panel, pos, codes, L, per_gap=per_gap, **kw)
    # the same call in a context whose budget just holds what one pass needs
    p = N.default_params(num_states=L, ne=20000, transition_mode=N.TRANS_PER_GAP if per_gap else N.TRANS_MATRIX0, **kw)
    from swiftimpute_b200.engine import Engine
    with Engine(0) as wide:
        wide.upload_panel(panel); wide.set_map(pos); wide.pbwt_build()
        wide.impute(codes, p, hap_prob=True)
        used, _ = wide.memory()  # without the segments' ends, which make room for any other allocation
    lmax = next(x for x in (4, 8, 16, 32) if L <= x)
    c = C or (16 if lmax == 32 else 32)
    one = (max(-(-M // c) - 1, 1) * lmax * B * 4 + 255) // 256 * 256  # the one pass' own checkpoints
    with Engine(0, hbm_budget_bytes=max(used + one, 1 << 20)) as tight:
        tight.upload_panel(panel); tight.set_map(pos); tight.pbwt_build()
        one_pass = tight.impute(codes, p, hap_prob=True)
    for key in got:
        assert np.array_equal(got[key], one_pass[key]), key


# per-target slots: rows staged in shared memory (up to 10,880 haplotypes) and read where they lie, lengths
# around the staged blocks (4) and code chunks (32), targets around a warp
@pytest.mark.parametrize("N_,M,B,L", [(2, 5, 3, 4), (33, 1, 1, 2), (300, 7, 31, 8), (300, 8, 32, 8), (300, 9, 33, 32),
                                      (1024, 65, 40, 16), (10880, 20, 5, 8), (10881, 20, 34, 8)])
def test_target_walk(engine, N_, M, B, L):
    panel, pos, _ = synth.make_panel(M, N_, 8, seed=M + N_)
    rng = np.random.default_rng(N_)
    codes = rng.integers(0, 5, (B, M)).astype(np.uint8)
    engine.upload_panel(panel)
    engine.set_map(pos)
    engine.pbwt_build(store_index=True)
    got = engine.select_states_target(L, codes)
    prefix = engine.prefix_rows()
    for b in range(B):
        assert np.array_equal(got[b], oracle.select_pairs_target(prefix, panel, codes[b], L)), b


# a batch's last target beside lanes without one: its slots are its own walk's, not those of a target without
# calls (what such a lane's codes read as), alone, at the end of a batch of any size and in the oracle
@pytest.mark.parametrize("N_", [300, 1024, 10880])
@pytest.mark.parametrize("B", [1, 2, 31, 33, 40, 63, 65])
def test_target_walk_last_target(engine, N_, B):
    M, L = 70, 8
    panel, pos, _ = synth.make_panel(M, N_, 8, seed=B + N_)
    codes = np.random.default_rng(B).choice(np.array([0, 2], np.uint8), (B, M))  # every marker typed, homozygous
    engine.upload_panel(panel)
    engine.set_map(pos)
    engine.pbwt_build(store_index=True)
    prefix = engine.prefix_rows()
    want = oracle.select_pairs_target(prefix, panel, codes[-1], L)
    none = oracle.select_pairs_target(prefix, panel, np.full(M, 3, np.uint8), L)
    assert (want != none).any(axis=(1, 2)).mean() > 0.5  # the two walks part: a store of the other one would show
    got = engine.select_states_target(L, codes)
    assert np.array_equal(got[-1], want)
    assert np.array_equal(engine.select_states_target(L, codes[-1:])[0], want)
    p = N.default_params(num_states=L, ne=20000, selection_kind=N.SEL_TARGET)
    batch, alone = engine.impute(codes, p, hap_prob=True), engine.impute(codes[-1:], p, hap_prob=True)
    for key in batch:
        assert np.array_equal(batch[key][-1], alone[key][0]), key


# the index built from sorted segments (up to about 20,000 haplotypes) and from swept groups: segment counts
# around powers of two, a last segment of any length, passes of eight markers with a remainder, many equal
# haplotypes (long groups) and none
@pytest.mark.parametrize("M,N_", [(127, 100), (128, 100), (129, 33), (192, 2), (256, 1025), (257, 5), (320, 64),
                                  (1000, 1024), (9600, 300), (9472, 31), (200, 20000), (140, 27000)])
@pytest.mark.parametrize("p1", [0.02, 0.5])
def test_index_segments(engine, M, N_, p1):
    rng = np.random.default_rng(M + N_)
    panel = (rng.random((M, N_)) < p1).astype(np.uint8)
    panel[:, N_ // 2:] = panel[:, :N_ - N_ // 2]  # every haplotype twice: ties keep their order
    engine.upload_panel(panel)
    engine.pbwt_build(store_index=N_ <= 1025, row_hashes=True)
    rows, hashes = oracle.pbwt_build_packed(synth.pack_panel(panel), N_)[:2]
    assert np.array_equal(engine.row_hashes(), hashes)
    if N_ <= 1025:
        assert np.array_equal(engine.prefix_rows(), oracle.pbwt_build(panel))


def test_index_rebuilt_in_place():
    """The same panel's index built again keeps its buffers: selections follow the build, imputation under
    a new panel's index is the new one's, and kept buffers make room within the budget."""
    from swiftimpute_b200.engine import Engine
    M, N_ = 700, 600
    panel, pos, _ = synth.make_panel(M, N_, 20, seed=3, spacing=1000)
    other, _, _ = synth.make_panel(M, N_, 20, seed=4, spacing=1000)
    codes, _, _ = synth.make_targets(panel, 40, synth.typed_every(M, 9), seed=5)
    p = N.default_params(num_states=8, ne=20000)

    def results(eng):
        return eng.select_states(8), eng.select_states(4), eng.impute(codes, p, hap_prob=True)

    with Engine(0) as eng:
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        first = results(eng)
        peak = eng.memory()[0]
        for _ in range(2):
            eng.pbwt_build()
            again = results(eng)
            assert np.array_equal(first[0], again[0]) and np.array_equal(first[1], again[1])
            for key in first[2]:
                assert np.array_equal(first[2][key], again[2][key])
        eng.impute(codes, N.default_params(num_states=8, ne=20000, flags=N.IMPUTE_FULL_CHAIN))
        eng.upload_panel(other); eng.set_map(pos); eng.pbwt_build()
        fresh = results(eng)
    with Engine(0) as eng:
        eng.upload_panel(other); eng.set_map(pos); eng.pbwt_build()
        for a, b in zip(results(eng)[:2], fresh[:2]):
            assert np.array_equal(a, b)
    with Engine(0, hbm_budget_bytes=peak + (4 << 20)) as eng:  # the build's own scratch is 4 MB here at most
        eng.upload_panel(panel); eng.set_map(pos); eng.pbwt_build()
        for L in (4, 8, 16, 32):
            eng.select_states(L)
        eng.pbwt_build(store_index=True)  # 1.7 MB of prefix rows beside what is kept
        again = results(eng)
        assert np.array_equal(first[0], again[0])


# warps that share a window group (one target, a few) against one warp a group (many): the same bits, for
# windows of any size
@pytest.mark.parametrize("C", [1, 2, 3, 8])
@pytest.mark.parametrize("L", [4, 8, 32])
def test_window_parts(engine, C, L):
    M = 1500
    panel, pos, _ = synth.make_panel(M, 300, 20, seed=C, spacing=1000)
    codes_all, _, _ = synth.make_targets(panel, 700, np.arange(M), seed=C + 1, het_range=(0.0, 1.0))
    codes = own_sites(codes_all, np.random.default_rng(C).integers(300, M, 700), seed=C + 2)
    codes[:64] = np.where(np.arange(M) % 3 == 0, codes_all[:64], 3)  # two groups on one array
    engine.upload_panel(panel)
    engine.set_map(pos)
    engine.pbwt_build()
    p = N.default_params(num_states=L, ne=20000, checkpoint_interval=C)
    many = engine.impute(codes, p, hap_prob=True)
    for rows in ([0], [5, 6, 7], list(range(60, 100)), [699]):
        few = engine.impute(codes[rows], p, hap_prob=True)
        for key in few:
            assert np.array_equal(few[key], many[key][rows]), (key, rows)


# L = 16: three CTAs an SM for a large batch, two for a small one: the oracle's, and the same bits in both
@pytest.mark.parametrize("L", [12, 16])
@pytest.mark.parametrize("own", [False, True])
def test_third_cta(engine, L, own):
    M, B = 2000, 5000  # 1,250 CTAs
    panel, pos, _ = synth.make_panel(M, 200, 12, seed=L, spacing=1000)
    codes_all, _, _ = synth.make_targets(panel, 40, np.arange(M), seed=L + 1, het_range=(0.0, 1.0))
    few = np.where(np.arange(M) % 8 == 0, codes_all, 3).astype(np.uint8)
    if own:
        few = own_sites(codes_all, np.random.default_rng(L).integers(100, 400, 40), seed=L + 2)
    check(engine, panel, pos, few, L)
    many = few[np.arange(B) % 40]
    for kw, out in (({}, {}), ({}, {"dosage": False}), ({"sampling": N.SAMPLE_PHILOX}, {"hap_prob": True, "haps": False})):
        p = N.default_params(num_states=L, ne=20000, **kw)
        a, b = engine.impute(few, p, **out), engine.impute(many, p, **out)
        for key in a:
            assert np.array_equal(a[key][np.arange(B) % 40], b[key]), (key, kw)


# the most haplotypes whose index is built by sorting (24,811), one more, and 25 elements a thread (from 24,577)
@pytest.mark.parametrize("N_", [24576, 24577, 24811, 24812])
def test_index_largest_sorted(engine, N_):
    M = 190  # two segments, the second one with a remainder of eight markers
    rng = np.random.default_rng(N_)
    panel = (rng.random((M, N_)) < 0.1).astype(np.uint8)
    panel[:, N_ // 2:] = panel[:, :N_ - N_ // 2]
    engine.upload_panel(panel)
    engine.pbwt_build(row_hashes=True)
    assert np.array_equal(engine.row_hashes(), oracle.pbwt_build_packed(synth.pack_panel(panel), N_)[1])

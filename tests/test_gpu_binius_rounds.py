"""Where the sum-check prover changes its launches: the last rounds in one CTA (by lookups
and by table bytes) and the direct or table fold over GF(2^128), against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REF = [([0, 1, 2], 1), ([0], 2)]
WIDE_TERMS = [([0, 1, 2, 3, 4, 0], 9), ([4, 4], 1), ([], 7), ([2], 200), (list(range(5)) * 3, 255)]


@pytest.mark.parametrize("level,k,m,terms", [
    (3, 12, 3, REF), (3, 13, 3, REF), (3, 14, 3, REF), (3, 9, 5, WIDE_TERMS), (3, 11, 40, [([39], 1), ([0, 39], 5)]),
    (3, 1, 1, [([0], 1)]), (3, 7, 1, [([], 3)]), (7, 5, 3, REF), (7, 6, 3, REF), (7, 7, 3, REF),
    (7, 4, 5, WIDE_TERMS), (7, 8, 1, [([0], 1 << 100)])])
def test_tail_rounds_match_oracle(orc, level, k, m, terms):
    from zs_b200 import native
    es = 1 if level == 3 else 16
    rng = np.random.default_rng(900 + 13 * k + level + m)
    tables = rng.bytes(m * (1 << k) * es)
    seed = rng.bytes(3 * k) if k % 2 else None
    got = native.binius_prove_combination(8 if level == 3 else 128, tables, k, m, terms, seed)
    assert got == orc.binius_prove(level, tables, k, m, terms, seed)


@pytest.mark.parametrize("m,length", [(3, 43690), (3, 43692), (1, 2), (7, 18726)])
def test_fold128_either_way_matches_oracle(orc, m, length):
    import torch
    from zs_b200 import native
    rng = np.random.default_rng(m + length)
    cur = rng.bytes(m * length * 16)
    r = int.from_bytes(rng.bytes(16), "little")
    d_cur = torch.frombuffer(bytearray(cur), dtype=torch.uint8).to("cuda")
    d_next = torch.zeros(m * (length // 2) * 16, dtype=torch.uint8, device="cuda")
    d_scratch = torch.zeros(65536, dtype=torch.uint8, device="cuda")
    native.binius_fold_device(128, d_cur.data_ptr(), length, m, r, d_next.data_ptr(), d_scratch.data_ptr())
    torch.cuda.synchronize()
    assert bytes(d_next.cpu().numpy()) == orc.binius_fold(7, cur, length, m, r)


@pytest.mark.parametrize("over", [1, 2, 257])
def test_fold128_table_equals_direct(orc, over):
    """The most elements that the direct fold takes, and `over` more, which go through the
    multiply table: equal rows, and the rows past the line as the oracle has them."""
    import torch
    from zs_b200 import native
    half = 1 << 18
    rng = np.random.default_rng(over)
    cur = rng.bytes((half + over) * 32)
    r = int.from_bytes(rng.bytes(16), "little")
    d_cur = torch.frombuffer(bytearray(cur), dtype=torch.uint8).to("cuda")
    d_scratch = torch.zeros(65536, dtype=torch.uint8, device="cuda")
    outs = []
    for rows in (half, half + over):
        d_next = torch.zeros(rows * 16, dtype=torch.uint8, device="cuda")
        native.binius_fold_device(128, d_cur.data_ptr(), 2 * rows, 1, r, d_next.data_ptr(), d_scratch.data_ptr())
        torch.cuda.synchronize()
        outs.append(bytes(d_next.cpu().numpy()))
    assert outs[0] == outs[1][:16 * half]
    for lo, hi in ((0, 512), (half, half + over)):
        assert outs[1][16 * lo:16 * hi] == orc.binius_fold(7, cur[32 * lo:32 * hi], 2 * (hi - lo), 1, r)


@pytest.mark.parametrize("points", range(1, 9))
def test_fold_fused_round_at_every_point_count(orc, points):
    """2^18 rows over GF(2^8): the second round folds and takes its values with all points in
    registers. Four tables, one of which no term names."""
    from zs_b200 import native
    terms = [([0, 3, 1, 0, 3, 1, 0][:points - 1], 3)]
    if points > 1:
        terms.append(([1], 1))
    rng = np.random.default_rng(1100 + points)
    tables = rng.bytes(4 << 18)
    got = native.binius_prove_combination(8, tables, 18, 4, terms)
    assert got == orc.binius_prove(3, tables, 18, 4, terms)


@pytest.mark.parametrize("k,m", [(8, 20), (8, 21), (8, 40), (8, 41)])
def test_chunks_of_gf128_rounds(orc, k, m):
    """Chunks of 64 rows (up to 20 tables), of 32 (up to 40), and a launch of its own for the
    fold beyond: two tables are named by terms."""
    from zs_b200 import native
    rng = np.random.default_rng(1200 + m)
    tables = rng.bytes(m * 16 << k)
    terms = [([0, m - 1], 5), ([0], 1)]
    got = native.binius_prove_combination(128, tables, k, m, terms)
    named = tables[:16 << k] + tables[(m - 1) * 16 << k:]  # the others change nothing
    assert got == orc.binius_prove(7, named, k, 2, [([0, 1], 5), ([0], 1)])


@pytest.mark.parametrize("k,m,terms", [(18, 5, [([4, 4], 1 << 90)]), (14, 33, [([32], 3), ([0, 32], 7)])])
def test_gf128_fold_by_the_table(orc, k, m, terms):
    """More than 2^18 elements to fold: the multiply table's launch, with the challenge in device
    memory, before values with the points in registers (2^18 rows) or in CTAs of their own, and
    the fused rounds after. Verified over the tables that the terms name."""
    from zs_b200 import native
    rng = np.random.default_rng(1300 + k)
    tables = rng.bytes(m * 16 << k)
    claimed, rounds = native.binius_prove_combination(128, tables, k, m, terms)
    names = sorted({f for fs, _ in terms for f in fs})
    named = b"".join(tables[f * 16 << k:(f + 1) * 16 << k] for f in names)
    renamed = [([names.index(f) for f in fs], c) for fs, c in terms]
    assert orc.binius_verify(7, named, k, len(names), renamed, claimed, rounds)
    bad = bytearray(rounds)
    bad[len(bad) // 2] ^= 1
    assert not orc.binius_verify(7, named, k, len(names), renamed, claimed, bytes(bad))


@pytest.mark.parametrize("k,points", [(8, 5), (9, 8), (8, 9), (8, 17)])
def test_gf128_rounds_of_many_points(orc, k, points):
    """More than four points over GF(2^128): the fold has a launch of its own while the chunks of
    a fused round would not fill the SMs."""
    from zs_b200 import native
    rng = np.random.default_rng(1400 + points)
    tables = rng.bytes(2 * 16 << k)
    terms = [([(j * j) % 2 for j in range(points - 1)], 77), ([1], 1 << 70), ([], 5)]
    assert native.binius_prove_combination(128, tables, k, 2, terms) == orc.binius_prove(7, tables, k, 2, terms)


def test_gf128_fused_rounds_of_many_points(orc):
    """2^16 rows at six points: fused while the chunks fill the SMs, then not."""
    from zs_b200 import native
    tables = np.random.default_rng(1500).bytes(16 << 16)
    terms = [([0] * 5, 9), ([0], 1)]
    claimed, rounds = native.binius_prove_combination(128, tables, 16, 1, terms)
    assert orc.binius_verify(7, tables, 16, 1, terms, claimed, rounds)
    bad = bytearray(rounds)
    bad[16 * 6 + 3] ^= 1
    assert not orc.binius_verify(7, tables, 16, 1, terms, claimed, bytes(bad))

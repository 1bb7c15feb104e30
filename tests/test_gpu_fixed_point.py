"""The fixed-point trainers at values where their rounding and their scales can go wrong: exact halves on the grid, rows of
zeros, tiny and denormal rows, values beyond the int8 range and beyond 2^21 steps of a grid, extremes next to a power of
two, rows on one side of zero.  Bit for bit against the sequential oracle."""
import numpy as np
import pytest

from helpers import assert_bit_equal, random_problem

pytestmark = pytest.mark.gpu

KINDS = ["halves", "zeros", "zero_side", "tiny", "denormal", "mixed", "large", "powers", "negative"]


def factors(kind, rng, rows, k):
    x = (rng.standard_normal((rows, k)) * 0.2).astype(np.float32)
    if kind == "halves":
        return (np.round(x * 512) / 512 + np.float32(1 / 1024)).astype(np.float32)
    if kind == "zeros":
        return np.zeros_like(x)
    if kind == "zero_side":
        x[::2] = 0
        return np.abs(x)
    if kind == "tiny":
        return x * np.float32(1e-30)
    if kind == "denormal":
        return x * np.float32(1e-38)
    if kind == "mixed":
        return x * (10.0 ** rng.integers(-6, 2, (rows, 1))).astype(np.float32)
    if kind == "large":
        return x * np.float32(20)
    if kind == "negative":                    # the smallest magnitude may decide the scale
        return (-np.abs(1 + x / 40) * np.float32(0.5) ** rng.integers(0, 3, (rows, 1))).astype(np.float32)
    scale = np.float32(2.0) ** rng.integers(-8, 2, (rows, 1)).astype(np.float32)
    x = np.clip(x, -1, 1) * scale
    x[:, 0] = (scale * np.float32(127.5 / 128))[:, 0]                        # top / hi a power of two, exactly or by a few units
    x[:, 1] = -(scale * np.float32(128.5 / 128))[:, 0] * (1 + rng.integers(-3, 4, rows) * np.float32(2.0 ** -23))
    return x.astype(np.float32)


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("bits", (8, 12, 16, "afp"))
def test_extreme_values_bit_exact(mascot, oracle, k, kind, bits):
    if kind == "denormal" and bits in (12, 16):
        pytest.skip("the rule's own result: 0 times an infinite scale")
    lr = 1e-6 if kind in ("mixed", "large") else 1e-3         # slow enough not to diverge
    rng = np.random.default_rng(KINDS.index(kind))
    n_users, n_items, n = 61, 37, 1201
    R, _, _ = random_problem(rng, n_users, n_items, n, k)
    P, Q = factors(kind, rng, n_users, k), factors(kind, rng, n_items, k)
    afp = bits == "afp"
    cfg = mascot.default_config(version=mascot.V_AFP if afp else mascot.V_MUPPET, k=k, deterministic=1, shuffle=0, epoch=50, learning_rate=lr,
                                decay=0.1, lam=0.05, muppet_width=0 if afp else bits, sample_ratio=0.1)
    with mascot.Engine(cfg) as eng:
        eng.set_ratings(R, R[:10], n_users, n_items)
        eng.set_factors(P, Q)
        eng.train_epoch(0)
        Pg, Qg = eng.get_factors(0)
    rules, lrs = oracle.rules_reference(), float(np.float32(lr))
    if afp:
        oracle.afp_run(k, R, None, P, Q, lrs, 0.05, 0, int(np.float32(n) / np.float32(10.0)), rules)
    else:
        oracle.muppet_run(k, R, None, P, Q, lrs, 0.05, bits, bits, rules, first_sample_pos=n - int(np.float32(n) * np.float32(0.1)))
    assert np.isfinite(P).all()
    assert_bit_equal(Pg, P, "P")
    assert_bit_equal(Qg, Q, "Q")


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("workers,n", [(40, 20011), (200, 20011), (700, 33000), (2500, 33000)])
def test_afp_workers_alone_and_together_in_their_warps(mascot, oracle, k, workers, n):
    """Several AFP workers, alone in a warp or not, on ratings that share no row: worker w takes the first run of 8 chunks
    number w in order, with a format state of its own."""
    rng = np.random.default_rng(workers)
    R, P, Q = random_problem(rng, n, n, n, k)
    R["u"], R["i"] = rng.permutation(n), rng.permutation(n)
    cfg = mascot.default_config(version=mascot.V_AFP, k=k, num_workers=workers, plain_user_stores=1, seed=3, epoch=50, learning_rate=0.01, decay=0.1, lam=0.05)
    with mascot.Engine(cfg) as eng:
        eng.set_ratings(R, R[:10], n, n)
        eng.set_factors(P, Q)
        order = eng.stream_order()
        w = eng.train_epoch(0).workers
        Pg, Qg = eng.get_factors(0)
    threshold = int(np.float32((n + w - 1) // w) / np.float32(10.0))
    run = 8 * (k // 8)
    assert w >= workers and n <= w * run, "only the first static runs"
    for b in range(0, n, run):
        oracle.afp_run(k, R[order[b:b + run]].copy(), None, P, Q, 0.01, 0.05, 0, threshold, oracle.rules_reference())
    assert_bit_equal(Pg, P, "P")
    assert_bit_equal(Qg, Q, "Q")


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("bits", (8, 12, 32))
@pytest.mark.parametrize("kind", ("mixed", "powers", "negative"))
def test_muppet_workers_side_by_side(mascot, oracle, k, bits, kind):
    """Two or four MuPPET workers in a warp, whose rows need different scales and some of them the exact formula: ratings that
    share no row, so that their order does not matter."""
    n = 20011
    rng = np.random.default_rng(k + bits)
    R, _, _ = random_problem(rng, n, n, n, k)
    R["u"], R["i"] = rng.permutation(n), rng.permutation(n)
    P, Q = factors(kind, rng, n, k), factors(kind, rng, n, k)
    cfg = mascot.default_config(version=mascot.V_MUPPET, k=k, num_workers=200, plain_user_stores=1, epoch=50, learning_rate=1e-6, decay=0.1, lam=0.05,
                                muppet_width=bits, sample_ratio=0.1)
    with mascot.Engine(cfg) as eng:
        eng.set_ratings(R, R[:10], n, n)
        eng.set_factors(P, Q)
        eng.train_epoch(0)
        Pg, Qg = eng.get_factors(0)
    oracle.muppet_run(k, R, None, P, Q, float(np.float32(1e-6)), 0.05, bits, bits, oracle.rules_reference(), first_sample_pos=n)
    assert_bit_equal(Pg, P, "P")
    assert_bit_equal(Qg, Q, "Q")

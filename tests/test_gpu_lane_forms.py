"""Workers of K/4 lanes (four elements each) and of K/8 lanes (eight), on both sides of the launch rule: ratings few enough for
the first run of one worker, in which rows come back at once, so that the sequential oracle has every bit of the result
and of the sampled statistics."""
import re

import numpy as np
import pytest

from helpers import assert_bit_equal, random_problem
from test_gpu_parity import assert_within_one_ulp
from test_gpu_update_edges import oracle_epoch, promoted_model

pytestmark = pytest.mark.gpu

# workers -> form: 1 to 8 (k=64: 16) of a single block are narrow; 9 to 16 (17 to 32), which fit a single block of the wide form only,
# and grids with few runs a worker are wide
WORKERS = (2, 8, 12, 16, 31, 300, 60000)


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("workers", WORKERS)
@pytest.mark.parametrize("version", ["sgd", "mpt", "memquant", "muppet8", "muppet12", "muppet32", "afp"])
def test_both_lane_forms_follow_the_oracle(mascot, oracle, k, workers, version):
    for n_users, n_items, n in ((1, 1, 9), (3, 2, k // 2 + 1), (17, 5, k)):
        R, P, Q = random_problem(np.random.default_rng(n + n_users), n_users, n_items, n, k, scale=0.2)
        muppet = version.startswith("muppet")
        v = dict(sgd=mascot.V_SGD, mpt=mascot.V_MPT, memquant=mascot.V_MEMQUANT, afp=mascot.V_AFP).get(version, mascot.V_MUPPET)
        width = int(version[6:]) if muppet else 0
        cfg = mascot.default_config(version=v, k=k, num_workers=workers, plain_user_stores=1, shuffle=0, epoch=50, learning_rate=0.01, decay=0.1, lam=0.05,
                                    muppet_width=width, sample_ratio=0.3)
        with mascot.Engine(cfg) as eng:
            eng.set_ratings(R, R[:1], n_users, n_items)
            eng.set_factors(P, Q)
            w = eng.train_epoch(0).workers
            Pg, Qg = eng.get_factors(0)
            gp, _, norms, _ = eng.sample_stats()
        rules = oracle.rules_reference()
        if muppet:
            first = n - int(np.float32(n) * np.float32(0.3))
            sums, norm = oracle.muppet_run(k, R, None, P, Q, float(np.float32(0.01)), 0.05, width, width, rules, first_sample_pos=first)
            if width != 32:
                assert_bit_equal(gp[:k], sums, "sum of gradients")
                assert_bit_equal(norms[:1], np.float32(norm), "sum of norms")
        elif version == "afp":
            oracle.afp_run(k, R, None, P, Q, 0.01, 0.05, 0, int(np.float32((n + w - 1) // w) / np.float32(10.0)), rules)
        else:
            P, Q = oracle_epoch(oracle, version, k, R, P, Q, 0.01, 0.05)
        assert_bit_equal(Pg, P, f"n {n} P")
        assert_bit_equal(Qg, Q, f"n {n} Q")


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("workers", WORKERS)
@pytest.mark.parametrize("users,items", [(False, False), (True, True), (True, False), (False, True)])
def test_both_lane_forms_of_the_precision_classes(mascot, oracle, k, workers, users, items):
    for n_users, n_items, n in ((1, 1, 9), (3, 2, k // 2 + 1), (17, 5, k)):
        R, P, Q = random_problem(np.random.default_rng(n + n_users), n_users, n_items, n, k, scale=0.2)
        cfg = mascot.default_config(version=mascot.V_MASCOT, k=k, num_workers=workers, plain_user_stores=1, shuffle=0, epoch=50, learning_rate=0.01, decay=0.1,
                                    lam=0.05, user_group_num=1, item_group_num=1, sample_ratio=0.3, interval=1, error_threshold=1e30)
        with mascot.Engine(cfg) as eng:
            eng.set_ratings(R, R[:1], n_users, n_items)
            eng.set_factors(P, Q)
            model, u2s, i2s = promoted_model(oracle, mascot, eng, k, P, Q, users, items)
            assert eng.train_epoch(5).error_check
            Pg, Qg = eng.get_factors(1)
            got = eng.sample_stats()
        Rs = R.copy()
        Rs["u"], Rs["i"] = u2s[R["u"]], i2s[R["i"]]
        lr = float(oracle.lr_schedule(0.01, 0.1, 50)[5])
        first = n - int(np.float32(n) * np.float32(0.3))
        want = model.run(Rs, None, lr, 0.05, oracle.rules_reference(), first_sample_pos=first, stats=True, item_stats_by_run=True)
        for a, b, what in zip(got, want, ("gsum_p", "gsum_q", "nsum_p", "nsum_q")):
            assert_bit_equal(a, b, f"n {n} {what}")
        Po, Qo = model.factors()
        assert_bit_equal(Pg, Po, f"n {n} P")
        assert_bit_equal(Qg, Qo, f"n {n} Q")


def narrow(k, runs):
    """(workers, ratings): a single block of narrow workers, or a grid of the fewest with `runs` runs of k ratings each - and 37 ratings more."""
    import torch
    workers = 2 * (128 // k) * torch.cuda.get_device_properties(0).multi_processor_count if runs else 8 * (128 // k)
    return workers, (runs or 5) * k * workers + 37


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("version", ["sgd", "mpt", "memquant", "muppet8", "muppet12", "afp"])
def test_many_runs_of_narrow_workers(mascot, oracle, k, version):
    """Ratings that share no row, in the hands of a single block - of MuPPET a grid of four runs a worker, the fewest that are narrow.
    AFP: two full runs a worker, which follow the oracle run by run."""
    muppet = version.startswith("muppet")
    workers, n = narrow(k, 4 if muppet else 0)
    if version == "afp":
        n = 2 * k * workers
    rng = np.random.default_rng(k)
    R, P, Q = random_problem(rng, n, n, n, k, scale=0.2)
    R["u"], R["i"] = rng.permutation(n), rng.permutation(n)
    v = dict(sgd=mascot.V_SGD, mpt=mascot.V_MPT, memquant=mascot.V_MEMQUANT, afp=mascot.V_AFP).get(version, mascot.V_MUPPET)
    width = int(version[6:]) if muppet else 0
    cfg = mascot.default_config(version=v, k=k, num_workers=workers, plain_user_stores=1, shuffle=0, epoch=50, learning_rate=0.01, decay=0.1, lam=0.05,
                                muppet_width=width, sample_ratio=0.0)
    with mascot.Engine(cfg) as eng:
        eng.set_ratings(R, R[:1], n, n)
        eng.set_factors(P, Q)
        assert eng.train_epoch(0).workers == workers
        Pg, Qg = eng.get_factors(0)
    rules = oracle.rules_reference()
    if muppet:
        oracle.muppet_run(k, R, None, P, Q, float(np.float32(0.01)), 0.05, width, width, rules, first_sample_pos=n)
    elif version == "afp":
        for w in range(workers):                        # runs w and w + workers, one after the other
            mine = np.concatenate([R[w * k:(w + 1) * k], R[(w + workers) * k:(w + workers + 1) * k]])
            oracle.afp_run(k, mine, None, P, Q, 0.01, 0.05, 0, int(np.float32((n + workers - 1) // workers) / np.float32(10.0)), rules)
    else:
        P, Q = oracle_epoch(oracle, version, k, R, P, Q, 0.01, 0.05)
    assert_bit_equal(Pg, P, "P")
    assert_bit_equal(Qg, Q, "Q")


@pytest.mark.parametrize("k", (128, 64))
def test_a_grid_of_narrow_afp_workers(mascot, oracle, k):
    """Rows and ratings that are all alike are updated alike, whichever worker has them and whatever it has had before."""
    workers, n = narrow(k, 4)
    R, P, Q = random_problem(np.random.default_rng(k), 1, 1, 1, k, scale=0.2)
    many = np.repeat(R, n)
    many["u"] = many["i"] = np.arange(n)
    cfg = mascot.default_config(version=mascot.V_AFP, k=k, num_workers=workers, plain_user_stores=1, epoch=50, learning_rate=0.01, decay=0.1, lam=0.05)
    with mascot.Engine(cfg) as eng:
        eng.set_ratings(many, many[:1], n, n)
        eng.set_factors(np.repeat(P, n, 0), np.repeat(Q, n, 0))
        assert eng.train_epoch(0).workers == workers
        Pg, Qg = eng.get_factors(0)
    oracle.afp_run(k, R, None, P, Q, 0.01, 0.05, 0, int(np.float32((n + workers - 1) // workers) / np.float32(10.0)), oracle.rules_reference())
    assert_bit_equal(Pg, np.repeat(P, n, 0), "P")
    assert_bit_equal(Qg, np.repeat(Q, n, 0), "Q")


CLASSES = ["mascot_hh", "mascot_fh", "mascot_hf", "mascot_ff", "switch"]


@pytest.mark.parametrize("k,runs,plain_stores,version", [(k, 0, s, v) for k in (128, 64) for s in (1, 0) for v in CLASSES]
                         + [(64, 16, 0, "mascot_hh"), (64, 16, 1, "mascot_fh")])
def test_many_runs_of_narrow_workers_of_the_precision_classes(mascot, oracle, k, runs, plain_stores, version):
    """Rows that one lane fetches and another one reads, over whole runs, tickets of the shared counter and both ways of
    writing user rows back: ratings that share no row, bit for bit, or within an ulp of the user rows where these are reductions of a
    change.  A single block, and grids of 16 runs a worker, the fewest that are narrow."""
    workers, n = narrow(k, runs)
    rng = np.random.default_rng(k)
    R, P, Q = random_problem(rng, n, n, n, k, scale=0.2)
    R["u"], R["i"] = rng.permutation(n), rng.permutation(n)
    cfg = mascot.default_config(version=mascot.V_SWITCH_ONLY if version == "switch" else mascot.V_MASCOT, k=k, num_workers=workers, plain_user_stores=plain_stores,
                                epoch=50, learning_rate=0.01, decay=0.1, lam=0.05, user_group_num=1, item_group_num=1, sample_ratio=0.0)
    with mascot.Engine(cfg) as eng:
        eng.set_ratings(R, R[:1], n, n)
        eng.set_factors(P, Q)
        if version != "switch":
            model, u2s, i2s = promoted_model(oracle, mascot, eng, k, P, Q, version[7] == "f", version[8] == "f")
        st = eng.train_epoch(0)
        assert st.workers == workers and st.updates == n
        Pg, Qg = eng.get_factors(0 if version == "switch" else 1)
    if version == "switch":
        P, Q = oracle_epoch(oracle, version, k, R, P, Q, 0.01, 0.05)
    else:
        Rs = R.copy()
        Rs["u"], Rs["i"] = u2s[R["u"]], i2s[R["i"]]
        model.run(Rs, None, 0.01, 0.05, oracle.rules_reference())
        P, Q = model.factors()
    if plain_stores:
        assert_bit_equal(Pg, P, "P")
    else:
        assert_within_one_ulp(Pg, P, version in ("mascot_hh", "mascot_hf", "switch"), "P")
    assert_bit_equal(Qg, Q, "Q")


def row_modes(call):
    """How the update kernels that `call` launches spread rows over lanes: ROWS_HALFQ = 3 and ROWS_F32Q = 4 are K/4 lanes a worker."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    names = [re.search(r"train_kernel<([^>]*)>", e.name) for e in prof.events()]
    modes = [re.sub(r"\([^)]*\)", "", m.group(1)).split(",")[2:4] for m in names if m]
    if not modes:
        pytest.skip("kernels cannot be traced here")
    return [int(x) for both in modes for x in both]


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("version,runs", [("sgd", 16), ("mpt", 16), ("memquant", 16), ("mascot", 16), ("muppet", 4), ("afp", 4)])
def test_lines_between_the_forms(mascot, k, version, runs):
    """Runs of k ratings a worker that make a grid narrow, sampled tails included, and the workers of a single block."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    grid = 2 * (128 // k) * sms
    v = dict(sgd=mascot.V_SGD, mpt=mascot.V_MPT, memquant=mascot.V_MEMQUANT, mascot=mascot.V_MASCOT, muppet=mascot.V_MUPPET, afp=mascot.V_AFP)[version]
    for workers, n, narrow_form in ((grid, runs * k * grid - 1, False), (grid, runs * k * grid, True), (8 * (128 // k), 4096, True), (8 * (128 // k) + 1, 4096, False)):
        R, P, Q = random_problem(np.random.default_rng(n), 3000, 2000, n, k)
        cfg = mascot.default_config(version=v, k=k, num_workers=workers, epoch=50, learning_rate=0.001, decay=0.1, lam=0.05, muppet_width=8 if version == "muppet" else 0,
                                    user_group_num=1, item_group_num=1, sample_ratio=0.05, interval=1, error_threshold=1e30)
        with mascot.Engine(cfg) as eng:
            eng.set_ratings(R, R[:1], 3000, 2000)
            eng.set_factors(P, Q)
            modes = row_modes(lambda: eng.train_epoch(10))
        assert len(modes) == 2 * (2 if version in ("mascot", "muppet") else 1), "plain launch and sampled tail"
        assert [m in (3, 4) for m in modes] == [narrow_form] * len(modes)

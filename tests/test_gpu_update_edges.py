"""The update kernel where it can go wrong: stream lengths around chunks and rings, worker counts that leave lanes of a
warp without work, and streams in which every few ratings meet the same user or item again (rows that are being
written while their next copy is on its way).  Bit for bit against the sequential oracle."""
import numpy as np
import pytest

from helpers import assert_bit_equal, random_problem

pytestmark = pytest.mark.gpu


def oracle_epoch(oracle, version, k, R, P, Q, lr, lam):
    rules = oracle.rules_reference()
    if version == "memquant":
        P16, Q16 = oracle.f2h(P), oracle.f2h(Q)
        oracle.memquant_run(k, R, None, P16, Q16, lr, lam, rules)
        return oracle.h2f(P16), oracle.h2f(Q16)
    if version == "mpt":
        P, Q = oracle.h2f(oracle.f2h(P)), oracle.h2f(oracle.f2h(Q))
        oracle.mpt_run(k, R, None, P, Q, lr, lam, rules)
    elif version == "switch":
        P16, Q16 = oracle.f2h(P), oracle.f2h(Q)
        oracle.switching_run(k, R, None, P16, Q16, 0, lr, lam, rules, first_sample_pos=None)
        return oracle.h2f(P16), oracle.h2f(Q16)
    else:
        oracle.sgd_run(k, R, None, P, Q, lr, lam, rules)
    return P, Q


def engine(mascot, version, k, **kw):
    v = dict(sgd=mascot.V_SGD, mpt=mascot.V_MPT, memquant=mascot.V_MEMQUANT, switch=mascot.V_SWITCH_ONLY)[version]
    return mascot.Engine(mascot.default_config(version=v, k=k, epoch=50, learning_rate=0.01, decay=0.1, lam=0.05, **kw))


@pytest.mark.parametrize("version,k", [("sgd", 128), ("sgd", 64), ("mpt", 128), ("memquant", 64), ("switch", 128)])
@pytest.mark.parametrize("n_users,n_items", [(1, 1), (2, 1), (1, 5), (3, 2), (7, 7)])
def test_rows_that_come_back_at_once(mascot, oracle, version, k, n_users, n_items):
    for n in (1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 33, 129, 517):
        R, P, Q = random_problem(np.random.default_rng(n), n_users, n_items, n, k)
        eng = engine(mascot, version, k, deterministic=1, shuffle=0)
        eng.set_ratings(R, R[:1], n_users, n_items)
        eng.set_factors(P, Q)
        eng.train_epoch(0)
        Pg, Qg = eng.get_factors(0)
        eng.close()
        Po, Qo = oracle_epoch(oracle, version, k, R, P.copy(), Q.copy(), 0.01, 0.05)
        assert_bit_equal(Pg, Po, f"n {n} P")
        assert_bit_equal(Qg, Qo, f"n {n} Q")


@pytest.mark.parametrize("version,k", [("sgd", 128), ("sgd", 64), ("memquant", 128), ("mpt", 64)])
@pytest.mark.parametrize("workers", [2, 3, 5, 17, 33, 64, 2048])
def test_every_rating_once_at_any_length_and_worker_count(mascot, oracle, version, k, workers):
    """No two ratings share a row, so the result does not depend on the order; plain stores keep it exact."""
    for n in (1, 9, 16, 100, 1023, 2049, 8191):
        rng = np.random.default_rng(n)
        R, P, Q = random_problem(rng, n, n, n, k)
        R["u"], R["i"] = rng.permutation(n), rng.permutation(n)
        eng = engine(mascot, version, k, num_workers=workers, plain_user_stores=1, seed=n)
        eng.set_ratings(R, R[:1], n, n)
        eng.set_factors(P, Q)
        eng.train_epoch(0)
        Pg, Qg = eng.get_factors(0)
        eng.close()
        Po, Qo = oracle_epoch(oracle, version, k, R, P.copy(), Q.copy(), 0.01, 0.05)
        assert_bit_equal(Pg, Po, f"n {n} P")
        assert_bit_equal(Qg, Qo, f"n {n} Q")


def promoted_model(oracle, mascot, eng, k, P, Q, users, items):
    """Engine and oracle with every group of the given sides in fp32, and the maps from ids to sorted indices."""
    u2s, i2s = eng.index_maps()
    Ps, Qs = np.empty_like(P), np.empty_like(Q)
    Ps[u2s], Qs[i2s] = P, Q
    prec, groups = [], []
    for side, (n, on) in enumerate(((len(P), users), (len(Q), items))):
        end, p, _ = eng.group_info(side)
        groups.append(np.searchsorted(end, np.arange(n), side="left").astype(np.uint32))
        prec.append(np.zeros_like(p))
        for g in range(len(end) if on else 0):
            eng.promote_group(side, g)
    model = oracle.MascotModel(k, Ps, Qs, groups[0], groups[1], *prec)
    for name, on, p in (("u", users, prec[0]), ("i", items, prec[1])):
        for g in range(len(p) if on else 0):
            model.promote(name, g)
    return model, u2s, i2s


@pytest.mark.parametrize("k", (128, 64))
@pytest.mark.parametrize("users,items", [(True, True), (True, False), (False, True)])
def test_classes_with_fp32_rows_asked_for_more_workers_than_fit(mascot, oracle, k, users, items):
    """The launch that takes short rings: rows that come back at once in the hands of the one worker that the first eight chunks
    make, and ratings that share no row over many workers.  Plain stores, bit for bit."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n_users, n_items, n in ((1, 1, 9), (2, 1, 33), (1, 5, 64), (3, 2, 63), (7, 7, 64), (7, 7, k), (1, 1, 1), (4097, 4097, 4097), (8191, 8191, 8191)):
        R, P, Q = random_problem(np.random.default_rng(n + n_users), n_users, n_items, n, k)
        if n == n_users:
            rng = np.random.default_rng(n)
            R["u"], R["i"] = rng.permutation(n), rng.permutation(n)
        cfg = mascot.default_config(version=mascot.V_MASCOT, k=k, num_workers=60000, plain_user_stores=1, seed=n, epoch=50, learning_rate=0.01, decay=0.1,
                                    lam=0.05, user_group_num=1, item_group_num=1)
        with mascot.Engine(cfg) as eng:
            eng.set_ratings(R, R[:1], n_users, n_items)
            eng.set_factors(P, Q)
            model, u2s, i2s = promoted_model(oracle, mascot, eng, k, P, Q, users, items)
            order = eng.stream_order()
            workers = eng.train_epoch(0).workers
            Pg, Qg = eng.get_factors(1)
        # deep rings: 16 warps per SM, short ones: 24, of two workers each (k=64: four)
        assert workers > 20 * 2 * (128 // k) * sms
        Rs = R[order].copy()
        Rs["u"], Rs["i"] = u2s[Rs["u"]], i2s[Rs["i"]]
        model.run(Rs, None, 0.01, 0.05, oracle.rules_reference())
        Po, Qo = model.factors()
        assert_bit_equal(Pg, Po, f"n {n} P")
        assert_bit_equal(Qg, Qo, f"n {n} Q")

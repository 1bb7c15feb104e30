"""The resident stream with run windows is the encoding step's order (windows of 4096), stably sorted by item inside every run
window - at sizes around the windows, and again after the stream has been replaced."""
import numpy as np
import pytest

from helpers import random_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (2, 4097, 16384, 16385, 100003))
@pytest.mark.parametrize("version", ("sgd", "mascot"))
def test_run_windows_sort_the_encoded_order(mascot, n, version):
    n_users, n_items, window = 700, 301, 1 << 14
    R, _, _ = random_problem(np.random.default_rng(n), n_users, n_items, n, 64)
    orders, maps = [], None
    for log2 in (12, 14):
        cfg = mascot.default_config(version=mascot.V_SGD if version == "sgd" else mascot.V_MASCOT, k=64, num_workers=4096, seed=n, run_window_log2=log2,
                                    sample_ratio=1.0, user_group_num=5, item_group_num=4)
        with mascot.Engine(cfg) as eng:
            eng.set_ratings(R, R[:min(n, 50)], n_users, n_items)
            maps = eng.index_maps()
            order = eng.stream_order()
            eng.reload_train(R)
            assert (eng.stream_order() == order).all()
            orders.append(order)
    assert sorted(orders[0].tolist()) == list(range(n))
    # the engine shortens the windows where the sampled tail would span fewer than four; a window of 2^12 changes nothing
    limit = n // 4 if version == "mascot" else n + window
    w = window
    while w > 4096 and w > limit:
        w //= 2
    want = orders[0].copy()
    item = maps[1][R["i"]].astype(np.int64)
    for b in range(0, n, w if w > 4096 else n):
        if w > 4096:
            part = want[b:b + w]
            want[b:b + w] = part[np.argsort(item[part], kind="stable")]
    assert (orders[1] == want).all()


def in_windows(order, item, seg, window):
    """`order`, stably sorted by item inside every piece that segments and multiples of `window` cut it into."""
    want = order.copy()
    cuts = sorted(set(seg) | set(range(0, seg[-1], window)))
    for b, e in zip(cuts, cuts[1:]):
        want[b:e] = want[b:e][np.argsort(item[want[b:e]], kind="stable")]
    return want


@pytest.mark.parametrize("version,seg", [("sgd", [0, 8192, 40960, 100003]), ("sgd", [0, 16384, 16384, 36864]), ("sgd", [0, 4096, 4097]),
                                         ("mascot", [0, 65536, 135168, 200704, 270001]), ("sgd", [0, 5000, 100003])])
def test_run_windows_of_several_segments(mascot, version, seg):
    """At the set-up and after a reload; segments that begin off the encoding step's windows take the sort of the coded stream."""
    n_users, n_items, n, window = 700, 301, seg[-1], 1 << 14
    R, _, _ = random_problem(np.random.default_rng(n), n_users, n_items, n, 64)
    orders = []
    for log2 in (12, 14):
        cfg = mascot.default_config(version=mascot.V_SGD if version == "sgd" else mascot.V_MASCOT, k=64, num_workers=4096, seed=n, run_window_log2=log2,
                                    sample_ratio=1.0, user_group_num=5, item_group_num=4)
        with mascot.Engine(cfg) as eng:
            eng.set_ratings_sharded(R, seg, R[:50], n_users, n_items)
            item = eng.index_maps()[1][R["i"]].astype(np.int64)
            orders.append(eng.stream_order())
            eng.reload_train(R)
            assert (eng.stream_order() == orders[-1]).all()
    for b, e in zip(seg, seg[1:]):
        assert sorted(orders[0][b:e].tolist()) == list(range(b, e))
    assert (orders[1] == in_windows(orders[0], item, seg, window)).all()


def test_reload_after_a_streamed_epoch_keeps_its_pieces(mascot):
    """The pieces of a streamed epoch become the segments of the resident stream; a reload sorts each of them in run windows."""
    n_users, n_items, piece, window = 7001, 301, 8 << 20, 1 << 14
    n = piece + 12345
    R, P, Q = random_problem(np.random.default_rng(3), n_users, n_items, n, 64)
    orders = []
    for log2 in (12, 14):
        with mascot.Engine(mascot.default_config(version=mascot.V_SGD, k=64, num_workers=4096, run_window_log2=log2)) as eng:
            eng.set_ratings(R, R[:50], n_users, n_items)
            eng.set_factors(P, Q)
            item = eng.index_maps()[1][R["i"]].astype(np.int64)
            eng.train_epoch_streamed(0, R)
            streamed = eng.stream_order()
            eng.reload_train(R)
            orders.append(eng.stream_order())
            assert eng.train_epoch(1).updates == n
            assert eng.train_segment(2, 1).updates == n - piece
    assert (orders[0] == streamed).all()
    assert (orders[1] == in_windows(streamed, item, [0, piece, n], window)).all()


@pytest.mark.parametrize("seg,shuffle", [([0, 100003], 1), ([0, 5000, 5000, 40960, 60001], 1), ([0, 3001], 0), ([0, 1], 1)])
def test_classes_keep_the_order_before(mascot, seg, shuffle):
    """Inside a precision class the ratings stay in the order that they had before the partition, also after several promotions one
    after the other, after a reload (a new stream, partitioned once) and after a streamed epoch (whose piece is a stream of its own)."""
    n_users, n_items, n = 700, 301, seg[-1]
    R, P, Q = random_problem(np.random.default_rng(n), n_users, n_items, n, 64)
    cfg = mascot.default_config(version=mascot.V_MASCOT, k=64, num_workers=4096, shuffle=shuffle, sample_ratio=1.0, user_group_num=6, item_group_num=5)
    with mascot.Engine(cfg) as eng:
        eng.set_ratings_sharded(R, seg, R[:1], n_users, n_items)
        eng.set_factors(P, Q)
        rows = [m[ids] for m, ids in zip(eng.index_maps(), (R["u"], R["i"]))]
        ends = [eng.group_info(side)[0] for side in (0, 1)]

        def expected(order, cuts):
            fp32 = [eng.group_info(side)[1][np.searchsorted(ends[side], rows[side], side="left")] != 0 for side in (0, 1)]
            cls = 2 * fp32[0] + fp32[1]
            return np.concatenate([order[b:e][np.argsort(cls[order[b:e]], kind="stable")] for b, e in zip(cuts, cuts[1:])])

        coded = order = eng.stream_order()
        for side, group in ((0, len(ends[0]) - 1), (1, 0), (0, 0), (1, len(ends[1]) - 1)):
            eng.promote_group(side, min(group, len(ends[side]) - 1))
            order = expected(order, seg)
            assert (eng.stream_order() == order).all()
        eng.reload_train(R)
        order = expected(coded, seg)
        assert (eng.stream_order() == order).all()
        eng.promote_group(0, min(1, len(ends[0]) - 1))
        assert (eng.stream_order() == expected(order, seg)).all()
        eng.train_epoch_streamed(0, R)
        piece = eng.stream_order()
        for side, group in ((1, 1), (0, 2)):
            eng.promote_group(side, min(group, len(ends[side]) - 1))
            piece = expected(piece, [0, n])
        assert (eng.stream_order() == piece).all()


@pytest.mark.parametrize("version,parts", [("mascot", [64, 34, 17, 8.5, 8.5]), ("muppet", [8, 16, 32, 64, 12]), ("sgd", [64, 64, 4])])
def test_pieces_of_a_long_streamed_epoch(mascot, version, parts):
    """Beyond two pieces the first or the last ones are smaller (sizes in 64ths of a piece); each is a permutation of its own range, and all are trained."""
    n_users, n_items, n = 7001, 301, (8 << 20) // 64 * int(sum(parts)) + 77
    R, P, Q = random_problem(np.random.default_rng(4), n_users, n_items, n, 64)
    v = dict(mascot=mascot.V_MASCOT, muppet=mascot.V_MUPPET, sgd=mascot.V_SGD)[version]
    with mascot.Engine(mascot.default_config(version=v, k=64, num_workers=4096, learning_rate=1e-4)) as eng:
        eng.set_ratings(R[:1000], R[:50], n_users, n_items)
        eng.set_factors(P, Q)
        assert eng.train_epoch_streamed(0, R).updates == n
        order = eng.stream_order()
        sizes = [eng.train_segment(1, s).updates for s in range(len(parts))]
        with pytest.raises(mascot.MascotError):
            eng.train_segment(1, len(parts))
    assert sum(sizes) == n and all(abs(s - e * (8 << 20) / 64) <= 4096 for s, e in zip(sizes, parts))
    at = 0
    for s in sizes:
        assert at % 4096 == 0 and (np.bincount(order[at:at + s] - at, minlength=s) == 1).all()
        at += s

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

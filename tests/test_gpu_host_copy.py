"""Factor matrices of every size class of the staged host copies: below the direct limit, pieces of one thread, ragged
last pieces, several blocks of whole slots, host addresses off every boundary; and buffers kept from one set of
ratings for the next, larger or smaller."""
import ctypes
import subprocess
import sys

import numpy as np
import pytest

from helpers import assert_bit_equal, random_problem

pytestmark = pytest.mark.gpu


def unaligned(a, off):
    """The same values at an address `off` floats past an allocation."""
    raw = np.empty(a.size + off, np.float32)
    raw[off:] = a.reshape(-1)
    return raw[off:].reshape(a.shape)


@pytest.mark.parametrize("n_users,n_items,off", [(3, 2, 0), (511, 257, 1), (769, 1, 3), (4099, 1023, 5), (20011, 333, 7), (131072, 65537, 1), (150001, 70001, 9)])
def test_factors_go_in_and_come_out_unchanged(mascot, n_users, n_items, off):
    k = 64
    rng = np.random.default_rng(n_users)
    R, P, Q = random_problem(rng, n_users, n_items, 50, k)
    eng = mascot.Engine(mascot.default_config(version=mascot.V_SGD, k=k, deterministic=1, shuffle=0))
    eng.set_ratings(R, R, n_users, n_items)
    for _ in range(2):
        eng.set_factors(unaligned(P, off), unaligned(Q, off + 2))
        Pg, Qg = eng.get_factors(0)
        assert_bit_equal(Pg, P, "P")
        assert_bit_equal(Qg, Q, "Q")
        eng.release_scratch()
    eng.close()


def test_an_engine_takes_larger_and_smaller_ratings(mascot, oracle):
    k = 128
    eng = mascot.Engine(mascot.default_config(version=mascot.V_SGD, k=k, deterministic=1, shuffle=0, lam=0.05))
    for n_users, n_items, n in ((50, 40, 900), (3000, 2000, 20011), (60, 1, 33), (3000, 1999, 20001)):
        R, P, Q = random_problem(np.random.default_rng(n), n_users, n_items, n, k)
        eng.set_ratings(R, R[:17], n_users, n_items)
        eng.set_factors(P, Q)
        eng.train_epoch(0)
        oracle.sgd_run(k, R, None, P, Q, 0.01, 0.05, oracle.rules_reference())
        Pg, Qg = eng.get_factors(0)
        assert_bit_equal(Pg, P, "P")
        assert_bit_equal(Qg, Q, "Q")
    eng.close()


def test_what_is_kept_between_calls_can_be_given_back_without_an_engine(mascot):
    """A program that only evaluates, and one whose engines are gone: device memory and helper threads come back."""
    code = """
import importlib.util, os, sys
import numpy as np, torch
spec = importlib.util.spec_from_file_location("mascot_binding", sys.argv[1]); M = importlib.util.module_from_spec(spec); spec.loader.exec_module(M)
k, n_users, n_items, n = 64, 200_000, 50_000, 100_000
rng = np.random.default_rng(0)
P, Q = rng.random((n_users, k), np.float32), rng.random((n_items, k), np.float32)
R = np.empty(n, M.RATING)
R["r"], R["u"], R["i"] = 3, rng.integers(0, n_users, n), rng.integers(0, n_items, n)
free = lambda: torch.cuda.mem_get_info()[0]
threads = lambda: len(os.listdir("/proc/self/task"))
want = M.rmse_host(P, Q, R, k)
M.release_cached()
idle, alone = free(), threads()
for _ in range(2):
    assert M.rmse_host(P, Q, R, k) == want
    kept, helped = idle - free(), threads() - alone
    M.release_cached()
    assert kept > 48 << 20 and idle - free() < 4 << 20, (kept, idle - free())
    assert helped > 0 and threads() == alone, (helped, threads() - alone)
with M.Engine(M.default_config(version=M.V_SGD, k=k)) as eng:
    eng.set_ratings(R, R, n_users, n_items)
    eng.set_factors(P, Q)
    M.release_cached()                                 # under a living engine: nothing that it uses
    assert abs(eng.eval_rmse() - want) < 1e-5 * want
M.release_cached()
assert idle - free() < 32 << 20 and threads() == alone      # (less the code of the update kernel)
"""
    subprocess.run([sys.executable, "-c", code, mascot.__file__], check=True, timeout=300)


@pytest.mark.parametrize("version", ("sgd", "mascot"))
@pytest.mark.parametrize("window", (0, 1))
def test_item_rows_can_be_opened_by_another_process(mascot, version, window):
    """The driver gives out a handle for their addresses, which stay the same; the rows are the ones the engine goes on with."""
    k, n_users, n_items, n = 64, 300, 200, 5000
    R, P, Q = random_problem(np.random.default_rng(5), n_users, n_items, n, k)
    cuda, got = ctypes.CDLL("libcuda.so.1"), []
    for asked in (False, True):
        cfg = mascot.default_config(version=mascot.V_SGD if version == "sgd" else mascot.V_MASCOT, k=k, deterministic=1, shuffle=0, l2_item_window=window)
        with mascot.Engine(cfg) as eng:
            eng.set_ratings(R, R[:10], n_users, n_items)
            eng.set_factors(P, Q)
            eng.train_epoch(0)
            if asked:
                (p16, b16), (p32, b32) = eng.item_rows(0, n_items)
                assert (p16 != 0) == (version == "mascot") and p32 != 0 and b32 == 4 * n_items * k
                for p in filter(None, (p16, p32)):
                    handle = ctypes.create_string_buffer(64)
                    assert cuda.cuIpcGetMemHandle(handle, ctypes.c_uint64(p)) == 0
                assert eng.item_rows(1, 2)[1][0] == p32 + 4 * k
            eng.train_epoch(1)
            got.append(eng.get_factors(0))
    assert_bit_equal(got[0][0], got[1][0], "P")
    assert_bit_equal(got[0][1], got[1][1], "Q")

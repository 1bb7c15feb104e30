"""What a user of this library waits for, as cases that can be timed and compared.

A case is one pass of a program around libmascot, through the Python binding of its C ABI:

  train            an engine that holds its ratings trains some epochs, reads the test RMSE after each one and
                   takes the factors out: the main loop of `quantized_mf`, without the set-up before it
  job              the whole of it: engine created, ratings handed over, factors set, epochs with their RMSE (group
                   errors and promotions among them), factors taken out, engine destroyed
  stream           epochs over ratings that stay in pinned host memory (mascot_train_epoch_streamed)
  setup            new ratings and fresh factors for an engine: degree sort, groups, coded stream, initialisation
  evaluate_host    the RMSE of a saved model on host arrays, what `test_mf` does
  evaluate_device  the same on buffers that are on the GPU already

Ratings have the laws of the benchmark configurations (synth.py): popularity by Zipf or log-normal weights, no
(user, item) pair twice, values from rank-16 factors plus noise on the grid of the data set.  Training starts from
a model that already knows those factors, spread over all k elements and disturbed, and runs at the learning rates of
the later epochs (a job: of a model that is trained further on new ratings): training of several workers is not
reproducible bit for bit, and in the first epochs from random numbers it amplifies what the races leave, so that two
correct runs could not be compared.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

mascot = importlib.import_module("icdm-2021_mascot_b200.mascot")

TRUE_RANK = 16


def _case(name, kind, version, k, users, items, n, n_test, user_law, user_s, item_law, item_s, grid, epochs, first_epoch=0, promoted=0.0,
          threshold=1e30, workers=0, groups=100, deterministic=False):
    return dict(name=name, kind=kind, version=version, k=k, users=users, items=items, n=n, n_test=n_test, user_law=user_law, user_s=user_s,
                item_law=item_law, item_s=item_s, grid=grid, epochs=epochs, first_epoch=first_epoch, promoted=promoted, threshold=threshold,
                workers=workers, groups=groups, deterministic=deterministic)


def listed():
    return [
        # The headline configuration: 100M ratings of 480k users on 18k films, k=128, the trainer the library is for.
        _case("mascot_100m", "train", 1, 128, 480_189, 17_770, 100_480_507, 1_408_395, "lognormal", 1.2, "zipf", 1.2, "int", 8, 20),
        # A music set at a quarter of its size after precision switching: most popular groups of both sides are in
        # fp32, so ratings of all four precision classes are trained and the rows no longer fit in L2.
        _case("mascot_promoted_63m", "train", 1, 128, 250_247, 156_240, 63_200_068, 1_000_990, "zipf", 1.0, "zipf", 1.0, "hundred", 6, 20, 0.4),
        # The k=64 configuration: 20M half-star ratings.
        _case("mascot_k64_20m", "train", 1, 64, 162_541, 59_047, 20_000_000, 500_000, "zipf", 1.0, "zipf", 1.0, "half", 10, 20),
        # The smallest configuration, plain fp32 SGD: epochs of a fraction of a millisecond.
        _case("sgd_k64_800k", "train", 5, 64, 10_000, 5_000, 800_000, 200_000, "zipf", 1.0, "zipf", 1.0, "int", 20, 20),
        # Mixed-precision training with fp32 master rows, on the 8M-rating configuration.
        _case("mpt_8m", "train", 4, 128, 71_567, 10_681, 8_000_000, 400_000, "zipf", 0.9, "zipf", 1.1, "half", 6, 20),
        # The adaptive fixed-point trainer, a comparison every user of the trainers runs.
        _case("afp_4m", "train", 2, 128, 50_003, 9_001, 4_000_003, 200_000, "zipf", 0.9, "zipf", 1.1, "half", 4, 20),
        # MuPPET from engine creation to factors: its int8 passes and per-epoch statistics, with a set-up of 2M ratings.
        _case("muppet_job_2m", "job", 3, 128, 30_011, 7_003, 2_000_003, 100_000, "zipf", 0.9, "zipf", 1.0, "half", 6),
        # A whole MASCOT training on the 8M-rating configuration: set-up, group errors, promotions, factors.
        _case("mascot_job_8m", "job", 1, 128, 71_567, 10_681, 8_000_000, 2_000_000, "zipf", 0.9, "zipf", 1.1, "half", 10, 0, 0.0, 0.7),
        # Ratings that stay on the host and are streamed through the engine, three pieces and a remainder.
        _case("stream_k128_27m", "stream", 1, 128, 162_541, 59_047, 27_000_019, 500_000, "zipf", 1.0, "zipf", 1.0, "half", 2, 20),
        # New ratings for an engine: what comes before the first epoch, at a size where sorting and copying count.
        _case("setup_40m", "setup", 1, 128, 300_007, 30_011, 40_000_003, 1_000_003, "lognormal", 1.2, "zipf", 1.1, "int", 0),
        # Evaluation of a saved model from host arrays.
        _case("evaluate_host_2m", "evaluate_host", 5, 128, 71_567, 10_681, 1, 2_000_000, "zipf", 0.9, "zipf", 1.1, "half", 0),
        # The smallest call: a validation set of some thousand ratings against a model on the GPU.
        _case("evaluate_device_10k", "evaluate_device", 5, 64, 10_000, 5_000, 1, 10_007, "zipf", 1.0, "zipf", 1.0, "int", 0),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choices(["train", "job", "stream", "setup", "evaluate_host", "evaluate_device"], [50, 15, 10, 10, 7, 8])[0]
    k = rng.choice([64, 128])
    version = rng.choices([1, 2, 3, 4, 5, 7], [50, 8, 8, 10, 16, 8])[0]
    if kind == "train" and version == 3:
        version = 5                       # MuPPET's width depends on the epochs before: whole jobs only
    if kind == "stream" and version == 2:
        version = 1                       # AFP is not streamed
    if kind == "setup":
        version = rng.choice([1, 1, 5])
    deterministic = kind == "train" and rng.random() < 0.08
    most = 2_500_000 if version in (2, 3) else 12_000_000 if kind == "job" else 30_000_000
    n = logu(20_000, 60_000) if deterministic else logu(50_000, most)
    users = max(400, min(1_000_000, n // logu(20, 200)))
    items = max(200, min(600_000, int(users * rng.uniform(0.04, 0.8))))
    while n + n // 4 > 0.1 * users * items:       # at most a tenth of the matrix, as in every configuration
        users, items = users * 2 + 1, items + items // 2 + 1
    n_test = max(1000, n // rng.choice([5, 20, 50]))
    if kind.startswith("evaluate"):
        n, n_test = 1, logu(1000, 5_000_000)
    user_law = rng.choice(["zipf", "zipf", "lognormal"])
    epochs = {"train": rng.randint(4, 12), "job": rng.randint(7, 12), "stream": rng.randint(1, 3)}.get(kind, 0)
    return _case("", kind, version, k, users, items, n, n_test, user_law, rng.uniform(0.7, 1.0) if user_law == "zipf" else rng.uniform(0.8, 1.3),
                 "zipf", rng.uniform(0.8, 1.2), rng.choice(["int", "half", "hundred"]), epochs, 0 if kind == "job" else rng.randint(15, 38),
                 rng.choice([0.0, 0.0, 0.2, 0.5]) if kind == "train" and version == 1 and not deterministic else 0.0,
                 0.7 if kind == "job" else 1e30, rng.choice([0, 0, 0, 2048]), rng.choice([10, 100]), deterministic)


# ---- data ------------------------------------------------------------------------------------------------------
def _popularity(law, s, n, gen):
    if law == "zipf":
        w = torch.arange(1, n + 1, dtype=torch.float64, device="cuda").pow_(-s)
    else:
        w = torch.exp(torch.randn(n, generator=gen, device="cuda", dtype=torch.float64) * s)
    w = w[torch.randperm(n, generator=gen, device="cuda")]
    return torch.cumsum(w / w.sum(), 0)


def _ratings(case, gen):
    """(ratings [n + n_test, 3] int32 on the GPU: bits of the value, user, item; true factors of both sides)"""
    users, items, total = case["users"], case["items"], case["n"] + case["n_test"]
    cu, ci = _popularity(case["user_law"], case["user_s"], users, gen), _popularity(case["item_law"], case["item_s"], items, gen)
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    while keys.numel() < total:
        want = int((total - keys.numel()) * 1.2) + 1024
        u = torch.searchsorted(cu, torch.rand(want, generator=gen, device="cuda", dtype=torch.float64)).clamp_(max=users - 1)
        i = torch.searchsorted(ci, torch.rand(want, generator=gen, device="cuda", dtype=torch.float64)).clamp_(max=items - 1)
        keys = torch.unique(torch.cat([keys, u * items + i]))
    keys = keys[torch.randperm(keys.numel(), generator=gen, device="cuda")[:total]]
    pt = torch.randn(users, TRUE_RANK, generator=gen, device="cuda") * 0.3
    qt = torch.randn(items, TRUE_RANK, generator=gen, device="cuda") * 0.3
    rec = torch.empty(total, 3, dtype=torch.int32, device="cuda")
    for b in range(0, total, 1 << 24):
        u, i = keys[b:b + (1 << 24)] // items, keys[b:b + (1 << 24)] % items
        x = 3.0 + 2.5 * (pt[u] * qt[i]).sum(1) + 0.5 * torch.randn(u.numel(), generator=gen, device="cuda")
        if case["grid"] == "int":
            x = x.round().clamp_(1, 5)
        elif case["grid"] == "half":
            x = ((x * 2).round() / 2).clamp_(0.5, 5)
        else:                              # 0..100 in steps of ten, rescaled to 1..5
            x = ((x - 1) * 2.5).round().clamp_(0, 10) / 2.5 + 1
        rec[b:b + (1 << 24), 0] = x.view(torch.int32)
        rec[b:b + (1 << 24), 1] = u.to(torch.int32)
        rec[b:b + (1 << 24), 2] = i.to(torch.int32)
    return rec, pt, qt


def _model(case, pt, qt, gen):
    """fp32 factors whose product is 3 + 2.5 * true product, turned into all k elements, plus noise."""
    k = case["k"]
    turn = torch.linalg.qr(torch.randn(k, k, generator=gen, device="cuda"))[0][:TRUE_RANK + 1]
    out = []
    for t in (pt, qt):
        wide = torch.cat([t * math.sqrt(2.5), torch.full((t.shape[0], 1), math.sqrt(3.0), device="cuda")], 1)
        out.append(wide @ turn + 0.02 * torch.randn(t.shape[0], k, generator=gen, device="cuda"))
    return out


def _host(t):
    return t.cpu().numpy().view(np.uint32)


def _config(case, seed):
    return mascot.default_config(version=case["version"], k=case["k"], lam=0.015, learning_rate=0.002 if case["kind"] == "job" else 0.01, decay=0.1, epoch=50, sample_ratio=0.05, interval=2,
                                 error_threshold=case["threshold"], user_group_num=case["groups"], item_group_num=case["groups"],
                                 num_workers=case["workers"], seed=seed + 1, deterministic=int(case["deterministic"]),
                                 shuffle=0 if case["deterministic"] else 1)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    rec, pt, qt = _ratings(case, gen)
    P, Q = _model(case, pt, qt, gen)
    s = dict(case=case, kind=kind, users=case["users"], items=case["items"])
    if kind == "evaluate_device":
        s.update(P=P, Q=Q, test=rec[1:].contiguous())
        return s
    train, test = rec[:case["n"]], mascot.as_ratings(_host(rec[case["n"]:]))
    if kind == "evaluate_host":
        s.update(P=P.cpu().numpy(), Q=Q.cpu().numpy(), test=test)
        return s
    cfg = _config(case, seed)
    if kind == "stream":                   # pinned, as the entry point asks for
        s["pinned"] = torch.empty(case["n"], 3, dtype=torch.int32, pin_memory=True)
        s["pinned"].copy_(train)
        train = mascot.as_ratings(s["pinned"].numpy().view(np.uint32))
    else:
        train = mascot.as_ratings(_host(train))
    del rec
    s.update(cfg=cfg, train=train, test=test)
    if kind == "job":
        s.update(P=P.cpu().numpy(), Q=Q.cpu().numpy())
        return s
    s["engine"] = mascot.Engine(cfg)
    if kind == "setup":
        return s
    s["engine"].set_ratings(train, test, case["users"], case["items"])
    s["engine"].set_factors(P.cpu().numpy(), Q.cpu().numpy())
    if case["promoted"]:                   # the most popular groups are the first to be switched
        for side in (0, 1):
            groups = len(s["engine"].group_info(side)[0])
            for g in range(int(groups * (1 - case["promoted"])), groups):
                s["engine"].promote_group(side, g)
    if kind == "train":
        s["train"] = None                  # the engine has its own copy
    return s


# ---- one pass --------------------------------------------------------------------------------------------------
def _epochs(s, engine, train_epoch):
    rmse = []
    for e in range(s["case"]["first_epoch"], s["case"]["first_epoch"] + s["case"]["epochs"]):
        train_epoch(e)
        rmse.append(engine.eval_rmse())
    P, Q = engine.get_factors()
    return {"P": P, "Q": Q, "rmse": np.array(rmse)}


def run(s):
    kind = s["kind"]
    if kind == "train":
        return _epochs(s, s["engine"], s["engine"].train_epoch)
    if kind == "stream":
        return _epochs(s, s["engine"], lambda e: s["engine"].train_epoch_streamed(e, s["train"]))
    if kind == "job":
        with mascot.Engine(s["cfg"]) as engine:
            engine.set_ratings(s["train"], s["test"], s["users"], s["items"])
            engine.set_factors(s["P"], s["Q"])
            return _epochs(s, engine, engine.train_epoch)
    if kind == "setup":
        engine = s["engine"]
        engine.set_ratings(s["train"], s["test"], s["users"], s["items"])
        engine.init_factors()
        user_map, item_map = engine.index_maps()
        return {"user_map": user_map, "item_map": item_map, "order": engine.stream_order(), "rmse": engine.eval_rmse()}
    if kind == "evaluate_host":
        return mascot.rmse_host(s["P"], s["Q"], s["test"], s["case"]["k"])
    out = ctypes.c_double()
    rc = mascot.load().mascot_rmse_device(ctypes.c_void_p(s["P"].data_ptr()), ctypes.c_void_p(s["Q"].data_ptr()), ctypes.c_uint32(s["case"]["k"]),
                                          ctypes.c_void_p(s["test"].data_ptr()), ctypes.c_uint64(s["test"].shape[0]), ctypes.byref(out))
    if rc != mascot.OK:
        raise mascot.MascotError(rc, "mascot_rmse_device")
    return out.value


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def work(case):
    k, rows, n, n_test = case["k"], case["users"] + case["items"], case["n"], case["n_test"]
    model = 4.0 * rows * k                 # fp32 factors, in or out
    stored = rows * k * (2.0 if case["version"] in (1, 7) else 4.0)
    if case["kind"].startswith("evaluate"):
        touched = min(rows, 2 * n_test)
        return {"bytes": 4.0 * touched * k + 12.0 * n_test, "flops": 2.0 * k * n_test}
    if case["kind"] == "setup":            # ratings in, stream and order out, factors initialised, one evaluation
        return {"bytes": 12.0 * n + 16.0 * n + 24.0 * n_test + 2 * stored, "flops": 2.0 * k * n_test}
    # an epoch reads every rating and reads and writes every row once; dot product, two gradients, two steps: 12 k
    per_epoch = 12.0 * n + 2 * stored + 12.0 * n_test + stored
    total = case["epochs"] * per_epoch + model
    if case["kind"] == "job":
        total += 12.0 * n + 12.0 * n + 24.0 * n_test + model
    return {"bytes": total, "flops": case["epochs"] * (12.0 * k * n + 2.0 * k * n_test)}


def tolerance(case):
    if case["deterministic"] or case["kind"] == "setup":
        return "exact"                     # one worker in the caller's order, or whole numbers and counter-based factors
    if case["kind"].startswith("evaluate"):
        return {"rel": 1e-6}               # the order of the sum is part of the result
    # several workers update shared rows in no fixed order, over some hundred updates a row; binary16 rows show it most
    return {"rel": 1e-2 if case["version"] in (1, 7) else 5e-3, "max": 0.4}

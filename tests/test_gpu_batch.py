"""Batched factorisation of many uneven tensors in one CUDA graph per
iteration (planc_gpu_batch_*), checked member by member against single
contexts and the CPU oracle."""
import numpy as np
import pytest

from helpers import cp_tensor, init_factors, rel

pytestmark = pytest.mark.gpu


def _members(n=6, seed=40):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        dims = tuple(int(d) for d in rng.integers(20, 70, size=3))
        k = int(rng.choice([4, 8, 16]))
        X, _ = cp_tensor(dims, k, noise=0.01, seed=seed + i)
        out.append((X, init_factors(dims, k, seed=seed + 100 + i)))
    return out


@pytest.mark.parametrize("prec", ["fp64", "bf16"])
def test_batch_matches_single_contexts(gpu, oracle_lib, prec):
    members = _members()
    iters = 8
    with gpu.Batch(0, prec, nstreams=4) as b:
        for X, F0 in members:
            b.add(X.astype(np.float32) if prec != "fp64" else X, F0)
        errs = b.run("hals", iters)
        for i, (X, F0) in enumerate(members):
            Fb, lb = b.get_factors(i)
            with gpu.Context(0, prec) as c:
                c.set_tensor(X.astype(np.float32) if prec != "fp64" else X)
                c.set_factors(F0)
                e = c.run("hals", iters)
                Fc, lc = c.get_factors()
            assert rel(errs[i], e) < 1e-13
            assert all(rel(a, b_) < 1e-13 for a, b_ in zip(Fb, Fc))
            if prec == "fp64":
                Fo, lo, eo = oracle_lib.ntf_run(X, F0, "hals", iters)
                assert rel(errs[i], eo) < 1e-10


@pytest.mark.parametrize("prec", ["fp64", "bf16"])
def test_batch_autotune_keeps_results(gpu, prec):
    members = _members(n=5, seed=50)
    with gpu.Batch(0, prec, nstreams=4) as b:
        for X, F0 in members:
            b.add(X.astype(np.float32) if prec != "fp64" else X, F0)
        e_ref = b.run("hals", 4)
        for i, (X, F0) in enumerate(members):
            b.set_factors(i, F0)
        ms = b.autotune("hals", trials=2)
        assert ms > 0
        e_tuned = b.run("hals", 4)
    # a retuned split-K count reorders the tensor cores' FP32 sums (BF16)
    assert rel(e_tuned, e_ref) < (1e-10 if prec == "fp64" else 1e-5)


def _grouped_members():
    # uneven shapes and ranks, including a mode-0 size that is a multiple of
    # 128 (the right contraction then forms mode 0's multi-TTV itself) and a
    # rank above 32 (the 64-column instances of the grouped kernels)
    rng = np.random.default_rng(60)
    specs = [((128, 40, 30), 8), ((30, 35, 40), 40), ((64, 20, 90), 32)]
    specs += [(tuple(int(d) for d in rng.integers(20, 70, size=3)), int(rng.choice([4, 8, 16, 32])))
              for _ in range(5)]
    out = []
    for i, (dims, k) in enumerate(specs):
        X, _ = cp_tensor(dims, min(k, 8), noise=0.01, seed=70 + i)
        out.append((X.astype(np.float32), init_factors(dims, k, seed=170 + i)))
    return out


@pytest.mark.parametrize("prec,algo", [("bf16", "hals"), ("bf16", "mu"), ("bf16x2", "hals")])
def test_batch_grouped_phases_give_the_same_bits(gpu, prec, algo, monkeypatch):
    # one launch per phase for all members vs one launch per member: the same
    # kernel bodies and summation orders, so the same bits
    members = _grouped_members()
    iters = 4
    res = {}
    for grouped in ("1", "0"):
        monkeypatch.setenv("PLANC_GPU_BATCH_GROUPED", grouped)
        with gpu.Batch(0, prec, nstreams=4) as b:
            for X, F0 in members:
                b.add(X, F0)
            errs = b.run(algo, iters)
            res[grouped] = (errs, [b.get_factors(i) for i in range(len(members))])
    (e1, f1), (e0, f0) = res["1"], res["0"]
    assert np.array_equal(e1, e0)
    for (Fa, la), (Fb, lb) in zip(f1, f0):
        assert np.array_equal(la, lb)
        assert all(np.array_equal(a, b_) for a, b_ in zip(Fa, Fb))


@pytest.mark.parametrize("count,dims", [(64, (492, 487, 2)), (4, (560, 541, 3))])
def test_batch_tables_grow_with_the_members(gpu, count, dims):
    # the tile lists of tensors with this many rows (I_0 I_1) need more than
    # 16 KB of argument tables a member
    k = 4
    members = [cp_tensor(dims, k, noise=0.01, seed=80 + i)[0].astype(np.float32) for i in range(2)]
    F0 = [init_factors(dims, k, seed=180 + i) for i in range(2)]
    with gpu.Batch(0, "bf16", nstreams=4) as b:
        for i in range(count):
            b.add(members[i % 2], F0[i % 2])
        errs = b.run("hals", 2)
        last = b.get_factors(count - 1)
    for i in range(2):
        with gpu.Context(0, "bf16") as c:
            c.set_tensor(members[i])
            c.set_factors(F0[i])
            e = c.run("hals", 2)
            F, lam = c.get_factors()
        assert np.array_equal(errs[i::2], np.tile(e, (count // 2, 1)))
    assert np.array_equal(last[1], lam)
    assert all(np.array_equal(a, b_) for a, b_ in zip(last[0], F))


def _image_members(few):
    # last modes above 128 (two row tiles a CTA up to rank 32, several row
    # groups above), I_0 not a multiple of 64, I_1 not a multiple of 4
    specs = [((61, 55, 200), 16)] if few else [
        ((61, 54, 129), 8), ((59, 57, 200), 16), ((62, 53, 300), 20), ((66, 50, 256), 32),
        ((60, 55, 140), 40), ((65, 51, 128), 64), ((57, 58, 90), 4), ((63, 52, 513), 24),
        ((61, 53, 300), 12), ((58, 57, 257), 33), ((67, 49, 131), 30), ((70, 47, 2), 5)]
    out = []
    for i, (dims, k) in enumerate(specs):
        X, _ = cp_tensor(dims, min(k, 8), noise=0.01, seed=90 + i)
        out.append((X.astype(np.float32), init_factors(dims, k, seed=190 + i)))
    return out


@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("prec", ["bf16", "bf16x2"])
def test_batch_long_contraction_gives_the_same_bits(gpu, prec, few, monkeypatch):
    # units of a split (few members) and of an eighth of a row group (many)
    # against the members' own launches
    members = _image_members(few)
    res = {}
    for grouped in ("1", "0"):
        monkeypatch.setenv("PLANC_GPU_BATCH_GROUPED", grouped)
        with gpu.Batch(0, prec, nstreams=4) as b:
            for X, F0 in members:
                b.add(X, F0)
            errs = b.run("hals", 3)
            res[grouped] = (errs, [b.get_factors(i) for i in range(len(members))])
    (e1, f1), (e0, f0) = res["1"], res["0"]
    assert np.array_equal(e1, e0)
    for (Fa, la), (Fb, lb) in zip(f1, f0):
        assert np.array_equal(la, lb)
        assert all(np.array_equal(a, b_) for a, b_ in zip(Fa, Fb))


@pytest.mark.parametrize("prec,algo", [("bf16", "hals"), ("bf16", "mu"), ("bf16", "anlsbpp"), ("fp64", "hals")])
def test_batch_runs_again_from_other_factors(gpu, prec, algo):
    # the captured iteration stays while new factors are set; a member's rank
    # changes, and changes back; other lengths
    members = _members(n=5, seed=210)
    data = [X.astype(np.float32) if prec != "fp64" else X for X, _ in members]
    starts = [F0 for _, F0 in members]

    def check(b, iters):
        errs = b.run(algo, iters)
        for i, X in enumerate(data):
            Fb, lb = b.get_factors(i)
            with gpu.Context(0, prec) as c:
                c.set_tensor(X)
                c.set_factors(starts[i])
                e = c.run(algo, iters)
                Fc, lc = c.get_factors()
            assert rel(errs[i], e) < 1e-13 and rel(lb, lc) < 1e-13
            assert all(rel(a, b_) < 1e-13 for a, b_ in zip(Fb, Fc))

    with gpu.Batch(0, prec, nstreams=4) as b:
        for X, F0 in zip(data, starts):
            b.add(X, F0)
        check(b, 4)
        for again, iters in enumerate((4, 7, 2)):
            for i, X in enumerate(data):
                k = 20 if (again, i) == (1, 1) else members[i][1][0].shape[1]
                starts[i] = init_factors(X.shape, k, seed=300 + 10 * again + i)
                b.set_factors(i, starts[i])
            check(b, iters)


@pytest.mark.parametrize("algo", ["hals", "mu"])
def test_batch_of_many_small_members_gives_the_same_bits(gpu, algo, monkeypatch):
    # enough rows of I_1 for four a CTA in the left multi-TTV, with remainders
    # of one, two and three
    members = []
    for i in range(26):
        dims, k = (20 + i, 46 + i % 7, 3 + i % 5), (4, 7, 16, 21, 32, 40)[i % 6]
        X, _ = cp_tensor(dims, 3, noise=0.01, seed=230 + i)
        members.append((X.astype(np.float32), init_factors(dims, k, seed=330 + i)))
    res = {}
    for grouped in ("1", "0"):
        monkeypatch.setenv("PLANC_GPU_BATCH_GROUPED", grouped)
        with gpu.Batch(0, "bf16", nstreams=4) as b:
            for X, F0 in members:
                b.add(X, F0)
            errs = b.run(algo, 3)
            res[grouped] = (errs, [b.get_factors(i) for i in range(len(members))])
    (e1, f1), (e0, f0) = res["1"], res["0"]
    assert np.array_equal(e1, e0)
    for (Fa, la), (Fb, lb) in zip(f1, f0):
        assert np.array_equal(la, lb)
        assert all(np.array_equal(a, b_) for a, b_ in zip(Fa, Fb))

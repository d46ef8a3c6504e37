"""The library's autotuner (adg_autotune): it times every elements-per-block
choice of the predictor on the context's own layout, restores the state,
keeps and records the fastest.  The choice changes the launch shape only:
tuned and default runs agree bit for bit, the tuned choice is the fastest
measured (never slower than the default), and a context created later with
elems_per_block = 0 takes the recorded choice."""
import numpy as np
import pytest

from parity import G, make_gpu_amr

pytestmark = pytest.mark.gpu


def run(s, n):
    s.advance(n, use_graph=True)
    return [s.get_U_w(l) for l in range(s.num_levels())]


def test_autotune_plain_is_bitwise_neutral_and_recorded(tmp_path, monkeypatch):
    monkeypatch.setenv("ADG_TUNE_CACHE", str(tmp_path / "tune.txt"))
    a = make_gpu_amr("kh_p3_amr", elems_per_block=16)
    b = make_gpu_amr("kh_p3_amr", elems_per_block=16)
    a.advance(2, use_graph=False)
    b.advance(2, use_graph=False)
    before = [b.get_U_w(l) for l in range(b.num_levels())]
    t0, step0 = b.time, b.step
    r = b.autotune(3)
    assert r["E"] in b.block_choices()["choices"]
    assert r["ms"][r["E"]] <= r["ms"][16]  # never slower than the default it replaces
    # the state, time and step count are as before the tuning
    assert b.time == t0 and b.step == step0
    for l, u in enumerate(before):
        assert np.array_equal(b.get_U_w(l), u)
    ua, ub = run(a, 8), run(b, 8)
    assert len(ua) == len(ub)
    for x, y in zip(ua, ub):
        assert np.array_equal(x, y)
    # recorded: a new context with elems_per_block = 0 takes the choice
    c = make_gpu_amr("kh_p3_amr")
    assert c.block_choices()["plain"] == r["E"]
    assert (tmp_path / "tune.txt").read_text().strip().endswith(f"plain {r['E']}")


def test_autotune_seeded_is_bitwise_neutral(tmp_path, monkeypatch):
    monkeypatch.setenv("ADG_TUNE_CACHE", str(tmp_path / "tune.txt"))
    seed = G.PredictorSeed(2, 3, hidden=128, rng_seed=3)
    a = make_gpu_amr("kh_p3_amr")
    b = make_gpu_amr("kh_p3_amr")
    for s in (a, b):
        seed.attach(s, mode=2, sweeps=2, tol=1e-3)
        s.advance(2, use_graph=False)
    r = b.autotune(2)
    assert b.block_choices()["seeded"] == r["E"]
    ua, ub = run(a, 6), run(b, 6)
    for x, y in zip(ua, ub):
        assert np.array_equal(x, y)


def _cached(tmp_path, monkeypatch, lines):
    """A context made with these lines of the cache file."""
    f = tmp_path / "tune.txt"
    f.write_text("".join(f"{k} {e}\n" for k, e in lines))
    monkeypatch.setenv("ADG_TUNE_CACHE", str(f))
    return make_gpu_amr("kh_p3_amr")


def _key(tmp_path, monkeypatch):
    """The key of the plain choice, as the library writes it."""
    monkeypatch.setenv("ADG_TUNE_CACHE", str(tmp_path / "key.txt"))
    make_gpu_amr("kh_p3_amr").autotune(1)
    return (tmp_path / "key.txt").read_text().split()[0]


def test_entries_of_other_kernels_or_sizes_are_not_taken(tmp_path, monkeypatch):
    """Some 700 elements, where the untuned choice is 8."""
    key = _key(tmp_path, monkeypatch)
    assert _cached(tmp_path, monkeypatch, [(key, 32)]).block_choices()["plain"] == 32
    # the key of builds whose plain path was the FP64 column kernel
    old = "/".join(key.split("/")[:5]) + "/plain"
    assert old.endswith("/D2P3/n16x16x1/L2/plain")
    assert _cached(tmp_path, monkeypatch, [(old, 32)]).block_choices()["plain"] == 8
    many = key.replace("/few/", "/many/")
    assert many != key
    assert _cached(tmp_path, monkeypatch, [(many, 32)]).block_choices()["plain"] == 8


@pytest.mark.parametrize("E", [8, 32])
def test_fp64_columns_do_not_take_the_plain_choice(tmp_path, monkeypatch, E):
    s = _cached(tmp_path, monkeypatch, [(_key(tmp_path, monkeypatch), E)])
    G.PredictorSeed(2, 3, hidden=128, rng_seed=3).attach(s, mode=1, sweeps=2, tol=1e-3)
    assert s.block_choices()["plain"] == E
    assert s.block_choices()["seeded"] == 16

"""Two handles on one GPU used by two threads: nothing in the API asks their callers to take turns, and neither may
change what the other's launches need."""
import threading

import numpy as np
import pytest

import rhydb_gpu as R
from rawtable import RawBuilder, oracle_for

pytestmark = pytest.mark.gpu

N = 3000


def partition(seed):
    """Two dictionary columns of 90 values: 8,281 combinations with the null groups (global counters), 91 and, with a
    position, 1,547 (counters in shared memory of different sizes)."""
    rng = np.random.default_rng(seed)
    seqs = ["".join(rng.choice(list("ACGT"), 40)) for _ in range(N)]
    b = RawBuilder(N).add_sequences("main", 0, "ACGT" * 10, seqs)
    for name in ("a", "b"):
        b.add_dict(name, [f"{name}{i:02d}" for i in rng.integers(0, 90, N)])
    raw = b.raw()
    t = R.Table.from_raw(raw)
    return t, R.Device(t, 0), oracle_for(t, raw), b


def nested(depth):
    """A filter whose program keeps about 2 * depth tiles on the stack."""
    q = "HasMut(main,1)"
    for i in range(depth):
        q = f"NOf(1,atleast,And({q},Or(HasMut(main,{i % 38 + 2}),SymEq(main,{i % 38 + 3},A))),And(HasMut(main,{i % 39 + 1}),HasMut(main,40)))"
    return q


def work(dev, kind, rounds):
    if kind == "calls":
        qs = [nested(d) for d in (1, 40, 3, 20)]
        return [dev.count(q) for _ in range(rounds) for q in qs]
    if kind == "batches":
        sets = [[nested(1)] * 2, [nested(3), nested(30)]]
        return [int(x) for _ in range(rounds) for qs in sets for x in dev.batch(qs)[0]]
    dims = [[("dict", 0)], [("dict", 0), ("seq", 0, 3)], [("dict", 0), ("dict", 1)]]
    return [tuple(c for _, c in dev.aggregate("True", d)[0]) for _ in range(rounds) for d in dims]


@pytest.mark.parametrize("kind,rounds", [("calls", 1500), ("batches", 400), ("aggregations", 400)])
def test_two_handles_in_two_threads(kind, rounds):
    tables = [partition(s) for s in (1, 2)]
    devs = [x[1] for x in tables]
    want = [work(d, kind, 1) for d in devs]  # alone
    if kind == "calls":
        assert want == [[x[2].count(nested(d)) for d in (1, 40, 3, 20)] for x in tables]
    got, errors = [None, None], []

    def run(i):
        try:
            got[i] = work(devs[i], kind, rounds)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for d in devs:
        d.close()
    assert not errors, errors
    assert got == [w * rounds for w in want]


def test_gradient_failure_stays_with_its_call():
    """One handle's bounded wait for the network's products gives up on every call (they are withheld, nothing is in
    flight); calls of another handle at the same time succeed, and every failed call reports it."""
    devs = [partition(s)[1] for s in (3, 4)]
    rng = np.random.default_rng(5)
    w = rng.normal(0, 0.1, R.MLP_NPARAM).astype(np.float32)
    x, t = rng.normal(size=(300, 24)).astype(np.float32), rng.normal(size=(300, 2)).astype(np.float32)
    want = devs[1].mlp_gradient(w, x, t)
    devs[0].test_withhold_copies(False, gradient=True)
    outcome = [[], []]

    def run(i):
        for _ in range(200):
            try:
                g, loss, y = devs[i].mlp_gradient(w, x, t)
                outcome[i].append(np.allclose(g, want[0], rtol=1e-4, atol=1e-6) and abs(loss - want[1]) <= 1e-5 * want[1])
            except R.RhyError as e:
                outcome[i].append("gave up" in str(e) and "failed")

    threads = [threading.Thread(target=run, args=(i,)) for i in (0, 1)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    devs[0].test_withhold_copies(False)
    after = devs[0].mlp_gradient(w, x, t)
    for d in devs:
        d.close()
    assert outcome[0] == ["failed"] * 200
    assert outcome[1] == [True] * 200
    assert np.allclose(after[0], want[0], rtol=1e-4, atol=1e-6)

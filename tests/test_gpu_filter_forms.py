"""The forms a filter leaf takes on the device, at the sizes where they can go wrong, against the oracle:
grouped row lists and their counters at every tile width, thresholds around the counters' sticky plane,
arrays stored as bitsets, the digits of the date index, the row lists of coverage leaves at the edges of
position blocks, and MutationProfiles on both sides of the limit between their two passes. Row sets and counts are equal bit for bit."""
import numpy as np
import pytest

import rhydb_gpu as R
from rawtable import RawBuilder, accession_table, oracle_for

pytestmark = pytest.mark.gpu


def check(dev, orc, queries):
    want = []
    for q in queries:
        bits, n = dev.compute_filter(q)
        obits, on = orc.compute_filter(q)
        assert n == on and np.array_equal(bits, obits), q
        want.append(on)
    counts, _ = dev.batch(queries)
    assert counts.tolist() == want
    return want


@pytest.fixture(scope="module")
def dense():
    """140,000 rows over few sites: bitsets, arrays on both sides of the dense limit, null rows, a
    ragged last chunk."""
    t = R.Table.generate(140000, seed=21, genome_len=600, pool_sites=120, n_aa_genes=2, null_fraction=0.01)
    dev = R.Device(t, 0)
    yield t, dev, oracle_for(t)
    dev.close()


@pytest.mark.parametrize("width", [4096, 8192, 16384, 32768, 65536])
def test_trees_at_every_tile_width(dense, width):
    t, dev, orc = dense
    qs = t.queries(40, seed=width, max_nof_children=24, max_leaves=48, use_aa=True, use_metadata=True)
    want = check(dev, orc, qs)
    own = R.Device(t, 0)  # set_tile_bits sets the widths of both paths
    own.set_tile_bits(width)
    assert check(own, orc, qs) == want
    own.close()
    counts, _ = dev.batch(qs, tile_bits=width)
    assert counts.tolist() == want


@pytest.mark.parametrize("children", [2, 3, 7, 8, 15, 16])
def test_thresholds_around_the_sticky_plane(dense, children):
    t, dev, orc = dense
    pos, chunk, sym, card, _ = t.containers(0)
    rows = {p: int(card[pos == p].sum()) for p in np.unique(pos)}
    common = sorted(rows, key=lambda p: -rows[p])[:children]  # the densest sites: counts pass every n
    qs = []
    for n in range(1, children):
        leaves = [f"HasMut(main,{p + 1})" for p in common]
        leaves[0] = f"Not({leaves[0]})"
        for kind in ("atleast", "exactly"):
            qs.append(f"NOf({n},{kind},{','.join(leaves)})")
            qs.append(f"NOf({n},{kind},{','.join(leaves[1:])},SymEq(main,{common[0] + 1},N))")
    check(dev, orc, qs)


@pytest.mark.parametrize("span", [0, 1, 127, 128, 16383, 16384, 2097151, 2097152])
def test_date_index_digits(span):
    n, base = 3000, 1000
    rng = np.random.default_rng(span)
    days = [None if i % 11 == 3 else base + int(rng.integers(0, span + 1)) for i in range(n)]
    days[0], days[1] = base, base + span
    b = RawBuilder(n).add_sequences("main", 0, "ACGT", ["ACGT"] * n).add_dates("date", days)  # owns raw's buffers
    raw = b.raw()
    t = R.Table.from_raw(raw)
    dev, orc = R.Device(t, 0), oracle_for(t, raw)
    ends = sorted({base - 1, base, base + 1, base + span // 2, base + span - 1, base + span, base + span + 1,
                   base + (span & 127), base + (span | 127), base + (span & ~127) - 1, base + 127, base + 128})
    qs = [f"DateBetween(date,{a},{b})" for a in ends for b in ends if a <= b]
    qs += [f"DateBetween(date,*,{b})" for b in ends] + [f"DateBetween(date,{a},*)" for a in ends]
    qs += [f"Not({q})" for q in qs[:20]] + [f"NOf(2,exactly,{qs[0]},{qs[-1]},{qs[len(qs) // 2]})"]
    check(dev, orc, qs)
    dev.close()


def test_coverage_lists_at_block_edges():
    b, raw, _ = accession_table(n_rows=3000, L=300, seed=9)
    t = R.Table.from_raw(raw)
    dev, orc = R.Device(t, 0), oracle_for(t, raw)
    qs = []
    for p in (1, 2, 19, 20, 126, 127, 128, 129, 130, 255, 256, 257, 281, 299, 300):
        c = t.local_reference(0)[p - 1]
        qs += [f"SymEq(main,{p},N)", f"SymEq(main,{p},{c})", f"Not(SymEq(main,{p},{c}))", f"Maybe(SymEq(main,{p},A))",
               f"Or(SymEq(main,{p},N),SymEq(main,{301 - p},{t.local_reference(0)[300 - p]}))",
               f"NOf(2,atleast,SymEq(main,{p},N),SymEq(main,{p},{c}),Not(SymEq(main,{301 - p},N)),HasMut(main,{p}))"]
    check(dev, orc, qs)
    dev.close()


@pytest.mark.parametrize("genome,rows,differences", [(600, 70000, 0), (600, 70000, 1), (600, 70000, 33), (600, 70000, 600),
                                                     (3000, 900, 2048), (3000, 900, 2049), (40000, 300, 2049)])
def test_profile_passes(genome, rows, differences):
    """Up to 2,048 positions off the local reference a profile is counted from its differences, above
    from the row index (terms in shared memory up to 32,767 positions, through the caches beyond)."""
    t = R.Table.generate(rows, seed=3, genome_len=genome, pool_sites=min(200, genome // 3), null_fraction=0.01)
    dev, orc = R.Device(t, 0), oracle_for(t)
    rng = np.random.default_rng(differences)
    ref = t.local_reference(0)
    seq = list(ref)
    for p in rng.choice(genome, differences, replace=False):
        seq[p] = "ACGT"["ACGT".index(seq[p]) - 1] if rng.random() < 0.8 else "N"
    seq = "".join(seq)
    off = sum(c != "N" and c != r for c, r in zip(seq, ref))
    short = f"MutProfileMutations(main,9,{1 + genome // 2}:A,{genome}:C)"
    qs = [f"MutProfile(main,{off + d},{seq})" for d in (0, 25)] + [short, f"And({short},HasMut(main,{genome // 2}))"]
    check(dev, orc, qs)
    dev.close()


@pytest.mark.parametrize("proportion,staged", [(0.0, False), (0.1, True), (1.0, True)])
def test_rows_of_the_final_pass(proportion, staged):
    """Mutations rows of a batch on both sides of its staging buffer (256 rows per slot over all slots), of
    nucleotide and amino-acid columns, with filters of no rows between them, in three position blocks."""
    t = R.Table.generate(3000, seed=12, genome_len=2500, pool_sites=1500, n_aa_genes=1, null_fraction=0.01)
    dev, orc = R.Device(t, 0), oracle_for(t)
    qs = t.queries(40, seed=13) + ["True", "And(True,Not(True))", "HasMut(main,1024)"]
    col = [i % 2 for i in range(len(qs))]
    want = [t.mutation_rows(c, orc.mutations(q, c)[0], proportion) for q, c in zip(qs, col)]
    n_rows = sum(map(len, want))
    assert (n_rows <= 256 * len(qs)) == staged
    for _ in range(2):  # the buffers of the first batch are taken again
        counts, rows, begin, cnt = dev.batch_rows(qs, [1] * len(qs), col, [proportion] * len(qs))
        got = [[(int(r["position"]), r["from_"].decode(), r["to"].decode(), int(r["count"]), int(r["coverage"]),
                 float(r["proportion"])) for r in rows[int(b):int(b) + int(n)]] for b, n in zip(begin, cnt)]
        assert got == want
    dev.close()


@pytest.mark.parametrize("children", [20, 60, 300])
def test_programs_around_the_launch_parameters(children):
    """Programs below and above 128 instructions (the launch's parameters, then device memory) alternate with
    short ones: count, row set and Mutations of one engine share the state that a call's end resets."""
    t = R.Table.generate(90000, seed=31, genome_len=900, pool_sites=400, null_fraction=0.01)
    dev, orc = R.Device(t, 0), oracle_for(t)
    long = "NOf(3,atleast," + ",".join(f"Or(HasMut(main,{2 * p + 1}),HasMut(main,{2 * p + 2}))" for p in range(children)) + ")"
    for q in (long, "HasMut(main,9)", long, "Not(HasMut(main,10))", "True"):
        obits, n = orc.compute_filter(q)
        assert dev.count(q) == n
        bits, m = dev.compute_filter(q)
        assert m == n and np.array_equal(bits, obits)
        counts, filtered = dev.mutations(q, 0)
        want, wn = orc.mutations(q, 0)
        assert filtered == wn == n and np.array_equal(counts, want)
    dev.close()


@pytest.fixture(scope="module")
def heavy_counts():
    """70,000 rows over 64 sites: containers of most rows of a chunk, missing intervals that start and end
    together, covered regions that end alone; and the oracle's Mutations by query."""
    n, L = 70000, 64
    rng = np.random.default_rng(8)
    ref = "ACGT" * (L // 4)
    rows = np.tile(np.frombuffer(ref.encode(), np.uint8), (n, 1))
    rows[rng.random(n) < 0.95, 20] = ord("N")
    rows[rng.random(n) < 0.4, 21:25] = ord("-")
    rows[rng.random(n) < 0.002, 40] = ord("T")
    rows[rng.random(n) < 0.45, 41] = ord("T")
    starts, ends = rng.integers(0, 10, n), rng.integers(L - 8, L + 1, n)
    at, some = np.arange(L), rng.random(n) < 0.03
    rows[some[:, None] & ((at < starts[:, None]) | (at >= ends[:, None]))] = ord("N")
    b = RawBuilder(n)
    b.add_sequences("main", 0, ref, [r.tobytes().decode() for r in rows])
    raw = b.raw()
    t = R.Table.from_raw(raw)
    dev, orc = R.Device(t, 0), oracle_for(t, raw)
    known = {}

    def mutations(q):
        if q not in known:
            known[q] = orc.mutations(q, 0)
        return known[q]

    yield dev, mutations
    dev.close()


@pytest.mark.parametrize("slots", [1, 12, 33, 65, 129, 257, 300])
def test_batched_counters(heavy_counts, slots):
    """The batched passes at one to eight mask words per row and at a second pass of one and two; the counters'
    planes fill up and are taken in between."""
    dev, mutations = heavy_counts
    forms = ["True", "Not(HasMut(main,41))", "SymEq(main,21,N)", "Not(SymEq(main,22,-))", "HasMut(main,42)"]
    qs = [f"And({forms[i % 5]},{forms[i // 5 % 5]})" for i in range(25)]
    qs = [qs[i * 7 % 25] for i in range(slots)]
    counts, muts = dev.batch(qs, [1] * slots, [0] * slots)
    for i, q in enumerate(qs):
        want, n = mutations(q)
        assert counts[i] == n and np.array_equal(muts[i], want), q


@pytest.mark.parametrize("differing", [True, False])
def test_mutations_around_the_row_index_limit(differing):
    """Filters of no rows, one, the most that take the row index, one more and all, one call after another, over
    a column with containers and one that equals its reference everywhere."""
    n = 70000
    rng = np.random.default_rng(4)
    pool = ["ACGTACGT", "ACGAACGT", "NCGTACG-", "ACNNNCGT"] if differing else ["ACGTACGT"]
    b = RawBuilder(n).add_sequences("main", 0, "ACGTACGT", [pool[i] for i in rng.integers(0, len(pool), n)])
    b.add_dates("date", list(range(n)))
    raw = b.raw()
    t = R.Table.from_raw(raw)
    dev, orc = R.Device(t, 0), oracle_for(t, raw)
    limit = dev.sparse_rows()[0]
    assert 1 < limit < n - 1
    for rows in (limit, limit + 1, 1, n, 0, limit + 1, limit):
        q = f"DateBetween(date,*,{rows - 1})" if rows else "And(True,Not(True))"
        counts, filtered = dev.mutations(q, 0)
        want, k = orc.mutations(q, 0)
        assert filtered == k == rows and np.array_equal(counts, want)
    dev.close()


@pytest.fixture(scope="module")
def container_forms():
    """140,000 rows: arrays of 1 to 4,096 rows around the narrow pass's steps, bitsets, and runs up to a whole
    chunk, a site each; and the oracle's Mutations by query."""
    n = 140000
    cards = [1, 15, 16, 17, 63, 64, 65, 239, 240, 241, 319, 320, 321, 959, 960, 961, 4095, 4096, 4097, 30000]
    spans = [(0, 65536), (65536, 131072), (10, 40000), (65530, 65540), (70000, 70033), (131072, 140000)]
    L = len(cards) + len(spans) + 1
    rng = np.random.default_rng(21)
    rows = np.full((n, L), ord("A"), np.uint8)
    for i, k in enumerate(cards):
        rows[rng.choice(65536, k, replace=False), i] = ord("C")
        rows[65536 + rng.choice(65536, k, replace=False), i] = ord("G")
    for i, (a, e) in enumerate(spans):
        rows[a:e, len(cards) + i] = ord("T")
    rows[rng.random(n) < 0.5, L - 1] = ord("C")
    b = RawBuilder(n)
    b.add_sequences("main", 0, "A" * L, [r.tobytes().decode() for r in rows])
    raw = b.raw()
    t = R.Table.from_raw(raw)
    dev, orc = R.Device(t, 0), oracle_for(t, raw)
    known = {}

    def mutations(q):
        if q not in known:
            known[q] = orc.mutations(q, 0)
        return known[q]

    yield dev, mutations, L
    dev.close()


@pytest.mark.parametrize("slots", [1, 15, 16, 17, 32, 33, 257, 289])
def test_narrow_container_pass(container_forms, slots):
    """Passes of one mask word (up to 32 queries, alone and after 256 others) and of two."""
    dev, mutations, L = container_forms
    forms = ["True", f"HasMut(main,{L})", f"Not(HasMut(main,{L}))", "HasMut(main,20)", f"Not(HasMut(main,{L - 1}))",
             "Not(HasMut(main,18))", "HasMut(main,21)", f"Or(HasMut(main,22),HasMut(main,{L}))"]
    qs = [f"Or({a},{b})" for a in forms for b in forms]
    qs = [qs[i * 11 % len(qs)] for i in range(slots)]
    dev.sparse_rows(batch=0)  # every filter takes the container pass
    counts, muts = dev.batch(qs, [1] * slots, [0] * slots)
    for i, q in enumerate(qs):
        want, n = mutations(q)
        assert counts[i] == n and np.array_equal(muts[i], want), q


@pytest.mark.parametrize("density", [0.0005, 0.3])
def test_resident_pass_under_capture(density):
    """The chain of dependent launches recorded into a CUDA graph, and replayed on another filter: the row index
    (few rows) and the dense passes."""
    torch = pytest.importorskip("torch")
    import ctypes
    t = R.Table.generate(100000, seed=17, genome_len=3000, pool_sites=500, null_fraction=0.01)
    dev = R.Device(t, 0)
    col = t.columns[0]
    rng = np.random.default_rng(3)
    rows = [np.concatenate([rng.random(t.n_rows) < density, np.zeros(t.n_chunks * R.CHUNK_ROWS - t.n_rows, bool)])
            for _ in range(2)]
    bits = [torch.from_numpy(np.packbits(r, bitorder="little").view(np.int32).copy()).cuda() for r in rows]
    f, n = torch.zeros_like(bits[0]), torch.zeros(1, dtype=torch.int64, device="cuda")
    counts = torch.empty(col.n_symbols, col.L, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(stream):
        dev.mutations_noalloc(0, f.data_ptr(), n.data_ptr(), counts.data_ptr(), status.data_ptr(),
                              ctypes.c_void_p(stream.cuda_stream))

    def load(i):
        f.copy_(bits[i])
        n.fill_(int(rows[i].sum()))
        torch.cuda.synchronize()  # the call below may run on the handle's own stream

    want = []
    for i in (0, 1):
        load(i)
        run(torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(counts.clone())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(torch.cuda.current_stream())
    for i in (1, 0, 0, 1):
        load(i)
        graph.replay()
        torch.cuda.synchronize()
        assert int(status) == 0 and torch.equal(counts, want[i])
    dev.close()

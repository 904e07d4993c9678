"""The resident Mutations pass is a chain of kernels whose launches overlap: each reads what the one before it wrote
only after waiting for it. Many passes in a row on one stream, without a wait of the host between them."""
import ctypes

import numpy as np
import pytest

import rhydb_gpu as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("column", [0, 1])
def test_passes_in_a_row_equal_passes_alone(column):
    torch = pytest.importorskip("torch")
    t = R.Table.generate(300000, seed=19, genome_len=9000, pool_sites=1500, n_aa_genes=2, null_fraction=0.01)
    dev = R.Device(t, 0)
    col = t.columns[column]
    rng = np.random.default_rng(6)
    stream = torch.cuda.Stream()
    filters = []
    for density in (0.3, 0.0, 1e-5, 1.0, 0.9, 1e-3):  # dense, no rows, the row index, all rows
        rows = np.zeros(t.n_chunks * R.CHUNK_ROWS, bool)
        rows[:t.n_rows] = rng.random(t.n_rows) < density
        bits = torch.from_numpy(np.packbits(rows, bitorder="little").view(np.int32).copy()).cuda()
        filters.append((bits, torch.tensor([int(rows.sum())], dtype=torch.int64, device="cuda")))
    order = rng.integers(0, len(filters), 120)
    tables = torch.full((len(order), col.n_symbols, col.L), -1, dtype=torch.int32, device="cuda")
    status = torch.zeros(len(order), dtype=torch.int32, device="cuda")
    alone = []
    torch.cuda.synchronize()

    def run(f, out, ok):
        dev.mutations_noalloc(column, f[0].data_ptr(), f[1].data_ptr(), out.data_ptr(), ok.data_ptr(),
                              ctypes.c_void_p(stream.cuda_stream))

    for f in filters:
        run(f, tables[0], status[0:1])
        torch.cuda.synchronize()
        alone.append(tables[0].clone())
    tables.fill_(-1)
    torch.cuda.synchronize()
    for i, k in enumerate(order):
        run(filters[k], tables[i], status[i:i + 1])
    torch.cuda.synchronize()
    assert not status.any()
    for i, k in enumerate(order):
        assert torch.equal(tables[i], alone[k]), (i, int(k))
    dev.close()


@pytest.mark.parametrize("mode", ["global", "relaxed"])
def test_prepared_profile_is_not_recorded(mode):
    """A single call's profile is copied from host memory that the next call reuses: recording it is refused in every
    capture mode. Programs without one are recorded and replayed."""
    torch = pytest.importorskip("torch")
    t = R.Table.generate(70000, seed=3, genome_len=3000, pool_sites=300)
    dev = R.Device(t, 0)
    stream = torch.cuda.Stream()
    ptr = ctypes.c_void_p(stream.cuda_stream)
    profile = "MutProfileMutations(main,4,241:T,1059:T,2100:G,2500:A)"
    assert dev.count(profile) > 0  # the buffers exist
    dev.plain_prepare([profile, "HasMut(main,9)"], [1, 1], [0, 0])
    with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream, capture_error_mode=mode):
        with pytest.raises(R.RhyError):
            dev.plain_launch(0, ptr)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
        dev.plain_launch(1, ptr)
    graph.replay()
    torch.cuda.synchronize()
    dev.plain_launch(0, ptr)  # and outside a capture
    torch.cuda.synchronize()
    dev.close()

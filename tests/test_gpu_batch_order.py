"""The order of a small batch's work items: the ones that begin last set the launch's end."""
import ctypes

import pytest

import rhydb_gpu as R

pytestmark = pytest.mark.gpu


def test_small_batch_starts_its_longest_programs_first():
    """40 filters over 2M rows are 1,240 items on 456 resident CTAs; tile by tile, the last tile of the longest
    program began after every other item and the launch took a sixth longer."""
    torch = pytest.importorskip("torch")
    t = R.Table.generate(2000000, seed=5, genome_len=1500, pool_sites=400)
    dev = R.Device(t, 0)
    stream = torch.cuda.Stream()
    ptr = ctypes.c_void_p(stream.cuda_stream)
    qs = sorted(t.queries(40, seed=3, max_depth=3, max_leaves=6), key=lambda q: -len(q))

    def filter_time(queries, **schedule):
        kept = dev.batch_schedule()
        dev.batch_schedule(**schedule)
        dev.batch_prepare(queries)
        dev.batch_schedule(**kept)
        dev.batch_launch(ptr, True, False)
        times = []
        for _ in range(40):
            a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            dev.batch_launch_parts(1, ptr)
            e.record(stream)
            e.synchronize()
            times.append(a.elapsed_time(e))
        return min(times)

    for _ in range(3):
        ordered = filter_time(qs, query_major=1)  # by hand: every tile of the longest first
        own = filter_time(qs[::-1])
        if own < 1.08 * ordered:
            break
    dev.close()
    assert own < 1.08 * ordered, (own, ordered)


def test_a_prepared_batch_is_copied_in_before_it_is_launched():
    torch = pytest.importorskip("torch")
    t = R.Table.generate(3000, seed=5, genome_len=1500, pool_sites=400)
    dev = R.Device(t, 0)
    for queries in (t.queries(3, seed=1), t.queries(60, seed=2)):
        want = [dev.count(q) for q in queries]
        dev.batch_prepare(queries)
        for call in (lambda: dev.batch_launch(None, False, True), lambda: dev.batch_launch_parts(1)):
            with pytest.raises(R.RhyError):
                call()
        dev.batch_launch(None, True, True)
        dev.batch_launch_parts(1)
        torch.cuda.synchronize()
        assert dev.batch_results(False)[0].tolist() == want
    dev.close()

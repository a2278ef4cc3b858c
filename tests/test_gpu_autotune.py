"""The default tuning sweep holds the untuned counts, and saved picks are those of this library's kernels."""
import json

import numpy as np
import pytest

from bbtc_b200 import Graph, autotune, graphs, options

pytestmark = pytest.mark.gpu


def median_ms(ctx, st, opts, torch, repeats=15):
    stream = torch.cuda.ExternalStream(ctx.stream)
    times = []
    with torch.cuda.stream(stream):
        for o in opts:
            st.count(opts=o)
        for _ in range(repeats):  # the options in turn, so that what else moves the time moves all of them
            row = []
            for o in opts:
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                st.count_async(opts=o)
                b.record(stream)
                st.count_wait()
                row.append(a.elapsed_time(b))
            times.append(row)
    return np.median(np.array(times), axis=0)


@pytest.mark.parametrize("kernel,scale", [("auto", 20), ("bitmap", 14), ("search", 14)])
def test_tuned_counts_are_not_slower(ctx, kernel, scale):
    torch = pytest.importorskip("torch")
    g = graphs.rmat(scale, 16, seed=1)
    st = Graph.from_csr(ctx, g, graphs.cuts(g, 8, "uni"))
    try:
        o, _ = autotune.sweep(st, base=options(kernel=kernel))
        plain, tuned = median_ms(ctx, st, [options(kernel=kernel), o], torch)
        assert tuned <= 1.1 * plain, (plain, tuned)  # two medians of one point differ by a few percent
    finally:
        st.free()


def test_picks_of_other_kernels_are_not_used(ctx, tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("BBTC_AUTOTUNE_CACHE", str(path))
    g = graphs.rmat(10, 8, seed=3)
    st = Graph.from_csr(ctx, g, graphs.cuts(g, 4, "uni"))
    try:
        saved = options(bitmap_words=2048, unit_work=8192, occupancy=8)
        # the key that picks of the tiled task rows were saved under: GPU and graph only
        key = f"{autotune.gpu_name(ctx.device)}|{autotune.graph_key(st)}"
        path.write_text(json.dumps({key: {"opts": {f: getattr(saved, f) for f, _ in saved._fields_}, "ms": 1.0}}))
        space = dict(bitmap_words=[512], warps_per_block=[8], unit_work=[256], occupancy=[4])
        o, ms = autotune.tune(st, **space)
        assert ms is not None and o.bitmap_words == 512
        o, ms = autotune.tune(st, **space)
        assert ms is None and o.bitmap_words == 512
        assert key in json.loads(path.read_text())  # another version's entries stay in the file
    finally:
        st.free()

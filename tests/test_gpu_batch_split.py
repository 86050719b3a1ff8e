"""Batch.capture and replay in split precision: the graph's slicing, tensor-core
and FP64 launches, with sectors on either side of the line between the two,
replayed on new elements, against the eager launch (bit for bit) and the FP64
product (the split form's 1e-13 of the norm)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(16, 200), (4, 40)])
def test_captured_split_batch(lo, hi):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu
    from trim_gb300 import workloads as wl

    pairs = wl.batched(24, lo, hi, 11)["pairs"]
    rng = np.random.default_rng(8)

    def tensors():
        out = []
        for specs in pairs:
            ts = []
            for s in specs:
                t = tu.UniTensor(s.bonds, s.labels)
                t.set_elem(rng.uniform(-1, 1, wl.elem_count(s.bonds)))
                ts.append(t)
            out.append(ts)
        return out

    first, second = tensors(), tensors()
    bt = tu.Batch([a for a, _ in first], [b for _, b in first])
    bt.capture("split")
    for ts in (first, second, first):
        for i, (a, b) in enumerate(ts):
            bt.put(i, a, b)
        bt.replay()
        tu.sync()
        got = [bt.output(i).get_elem() for i in range(len(ts))]
        bt.launch("split")
        tu.sync()
        for i, (a, b) in enumerate(ts):
            assert np.array_equal(got[i], bt.output(i).get_elem())
            want = tu.contract(a, b, mode="fp64").get_elem()
            assert np.linalg.norm(got[i] - want) <= 1e-13 * np.linalg.norm(want)

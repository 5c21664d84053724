"""fmcs_run_batch: many independent instances in one batch, each checked
against the oracle on its own rows (instance-local oids and group ids)."""
import numpy as np
import pytest

from fastmulticolsort_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [[8, 24, 40], [32, 40], [8, 64]])
def test_batch_matches_per_instance_oracle(ctx, split):
    rng = np.random.default_rng(sum(split))
    sizes = [1, 2, 3, 17, 129, 5000, 70000, 0, 1024, 4097, 12345, 1]
    sizes += list((2 ** rng.uniform(10, 16, size=20)).astype(int))
    total = int(sum(sizes))
    cols, bw = W.cols_uniform(total, [8, 24, 40], seed_index=5, distinct=[16, 0, 0])
    order = np.zeros(total, np.uint32)
    group = np.zeros(total, np.uint32)
    counts = ctx.run_batch(cols, bw, split, sizes, order, group)
    off = 0
    for k, n in enumerate(sizes):
        if n == 0:
            assert counts[k] == 0
            continue
        sub = [c[off:off + n].copy() for c in cols]
        o, g, ng = O.run_plan_sort(sub, bw, split)
        assert np.array_equal(order[off:off + n], o), k
        assert np.array_equal(group[off:off + n], g), k
        assert counts[k] == ng
        off += n


def test_batch_rejects_bad_instances(ctx):
    from fastmulticolsort_b200 import capi
    import ctypes
    cols, bw = W.cols_uniform(100, [8, 24], seed_index=6)
    L = capi.load()
    inst = (capi.Instance * 2)(capi.Instance(0, 50), capi.Instance(60, 40))   # gap: not contiguous
    ptrs = (ctypes.c_void_p * 2)(*[c.ctypes.data for c in cols])
    order = np.zeros(100, np.uint32)
    rc = L.fmcs_run_batch(ctx.handle, ptrs, capi._u32arr([2, 4]), capi._u32arr(bw), 2, capi._u32arr([32]), 1,
                          inst, 2, 100, order.ctypes.data, None, None)
    assert rc == capi.FMCS_E_INVAL


@pytest.mark.parametrize("shift", [0, 1, 3])
def test_batch_device_outputs_any_alignment(ctx, shift):
    """Device outputs that start on and off a 16-byte boundary, instance borders
    inside and at the ends of the 8,192-row steps, empty instances between."""
    import torch
    sizes = [8192, 0, 1, 8191, 3, 0, 0, 16381, 4096, 2, 40000, 0]
    total = int(sum(sizes))
    cols, bw = W.cols_uniform(total, [8, 24], seed_index=8, distinct=[3, 90])
    dev = [torch.from_numpy(c.view({2: np.int16, 4: np.int32}[c.itemsize])).cuda() for c in cols]
    order = torch.full((total + 8,), -7, dtype=torch.int32, device="cuda")
    group = torch.full((total + 8,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    counts = ctx.run_batch(dev, bw, [8, 24], sizes, order[shift:shift + total], group[shift:shift + total])
    h_order, h_group = order.cpu().numpy(), group.cpu().numpy()
    for a in (h_order, h_group):
        assert (a[:shift] == -7).all() and (a[shift + total:] == -7).all()
    off = 0
    for k, n in enumerate(sizes):
        if n:
            o, g, ng = O.run_plan_sort([c[off:off + n].copy() for c in cols], bw, [8, 24])
            assert np.array_equal(h_order[shift + off:shift + off + n].view(np.uint32), o), k
            assert np.array_equal(h_group[shift + off:shift + off + n].view(np.uint32), g), k
            assert counts[k] == ng
        off += n

"""The table of an ensemble's trees, made of CPU tensors (what it holds are addresses and sizes)."""
import pytest
import torch

from legateboost_b200.tree import TreeTable


def tree(M, K, leaf_type=torch.float64, split_type=torch.float64):
    return torch.arange(M * K).reshape(M, K).to(leaf_type), torch.full((M,), -1, dtype=torch.int32), torch.zeros(M, dtype=split_type)


def test_rows_hold_addresses_and_offsets():
    trees = [tree(7, 3), tree(1, 3), tree(15, 3)]
    t = TreeTable(trees)
    rows = t.table.numpy()
    off = 0
    for row, (lv, ft, sv) in zip(rows, trees):
        assert list(row[:3]) == [lv.data_ptr(), ft.data_ptr(), sv.data_ptr()]
        assert row[3] & 0xffffffff == len(ft) and row[3] >> 32 == off
        off += len(ft)
    assert (t.n_trees, t.n_outputs, t.max_nodes, t.total_nodes, t.reusable) == (3, 3, 15, 23, True)


@pytest.mark.parametrize("change", ["leaf type", "split type", "strided", "one dimension"])
def test_arrays_of_other_types_and_strides_are_copied(change):
    lv, ft, sv = tree(7, 1)
    if change == "leaf type":
        lv = lv.to(torch.float32)
    elif change == "split type":
        sv = sv.to(torch.float32)
    elif change == "strided":
        lv = torch.arange(14, dtype=torch.float64).reshape(7, 2)[:, :1]
    else:
        lv = lv[:, 0]
    t = TreeTable([tree(3, 1), (lv, ft, sv)])
    assert t.reusable == (change == "one dimension")
    for i, (kept, given) in enumerate(zip(t.keep[3:], (lv, ft, sv))):
        assert kept.is_contiguous() and torch.equal(kept, given.to(kept.dtype)) and t.table[1, i] == kept.data_ptr()
    assert not t.reusable or t.keep[3] is lv


def test_bad_ensembles_are_refused():
    lv, ft, sv = tree(7, 2)
    for bad in ([(lv[:6], ft, sv)], [(lv, ft, sv[:6])], [(lv, ft, sv), tree(7, 1)], [(lv[:0], ft[:0], sv[:0])]):
        with pytest.raises(ValueError):
            TreeTable(bad)

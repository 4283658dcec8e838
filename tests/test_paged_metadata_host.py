"""The native check of a paged call's metadata reads host memory, so it looks at the arrays before it does."""

import numpy as np
import pytest

from extensions_b200 import tiny_llm_ext_b200 as ext
from tiny_llm_b200.attention import validate_paged_metadata

TABLE = np.array([[3, 1, -1], [0, -1, -1]], dtype=np.int32)
CTX = np.array([20, 5], dtype=np.int32)


def clean(ctx, table):
    return ext.paged_metadata_clean(ctx, table, 16, 8, 1)


def test_whole_arrays():
    assert clean(CTX, TABLE)
    validate_paged_metadata(CTX, TABLE, 16, 8, 1)


@pytest.mark.parametrize("ctx,table", [
    (CTX[:1], TABLE), (np.concatenate([CTX, CTX]), TABLE), (CTX[None], TABLE), (CTX, TABLE[0]), (CTX[:0], TABLE),
    (CTX.astype(np.int64), TABLE), (CTX, TABLE.astype(np.int64)), (CTX, TABLE.astype(np.int16)), (CTX, np.asfortranarray(TABLE)), (np.repeat(CTX, 2)[::2], TABLE),
])
def test_arrays_that_are_not_read(ctx, table):
    assert not clean(ctx, table)


def test_fewer_lengths_than_rows_are_refused():
    with pytest.raises(IndexError):
        validate_paged_metadata(CTX[:1], TABLE, 16, 8, 1)


@pytest.mark.parametrize("table", [np.asfortranarray(TABLE), TABLE.astype(np.int64)])
def test_other_layouts_are_checked_all_the_same(table):
    validate_paged_metadata(CTX, table, 16, 8, 1)
    wrong = table.copy(order="K")
    wrong[1, 0] = 3
    with pytest.raises(ValueError, match="aliased"):
        validate_paged_metadata(CTX, wrong, 16, 8, 1)

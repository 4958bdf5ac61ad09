"""Saved tuning tables: a table comes back as it was written, and entries of older
tables whose index names another sort shape since are left out."""
import pytest

pytestmark = pytest.mark.gpu

NAME = "gbcompute_tuning.txt"
KEPT = {"sort:u32k:2^20": 6, "sort:u32kv:2^20": 7, "sort:u64k:2^20": 5, "segsort:u64kv:2^24:avg2^8": 4096,
        "segsort:u64kv:2^24:avg2^8:msd": 8}
RENAMED = {"sort:u32k:2^24": 7, "sort:u32k:2^28": 8, "sort:u32kv:2^24": 8, "sort:u64k:2^24": 6, "sort:u64kv:2^24": 6}


def test_older_tables(gbc, tmp_path):
    lines = ["# gbcompute tuning table: <op:dtype:size class[:distribution]> <variant>"]
    (tmp_path / NAME).write_text("\n".join(lines + [f"{k} {v}" for k, v in {**KEPT, **RENAMED}.items()]) + "\n")
    ctx = gbc.Context(cache_dir=str(tmp_path))
    assert {k: ctx.tuning_get(k) for k in KEPT} == KEPT
    assert all(ctx.tuning_get(k) == -1 for k in RENAMED)  # no entry
    ctx.close()


def test_a_table_comes_back(gbc, tmp_path):
    ctx = gbc.Context()
    for k, v in {**KEPT, **RENAMED}.items():
        ctx.tuning_set(k, v)
    ctx.tuning_save(str(tmp_path / NAME))
    ctx.close()
    ctx = gbc.Context(cache_dir=str(tmp_path))
    assert {k: ctx.tuning_get(k) for k in {**KEPT, **RENAMED}} == {**KEPT, **RENAMED}
    ctx.close()

"""Which form of a kernel a call takes: the rules that the library answers without a device."""

from ctypes import c_int
from types import SimpleNamespace

import torch

from strata_inference_b200.kernels import native


def _in_runs(rows, n_seqs, H, G, kd=128, taps=4):
    return bool(native.library().sib_delta_prepare_in_runs(*map(c_int, (rows, n_seqs, H, G, kd, taps))))


def test_delta_prepare_takes_runs_where_sequences_are_long_and_rows_are_many():
    for heads in ((8, 4), (16, 8), (4, 2), (16, 2)):
        assert not any(_in_runs(n, n, *heads) for n in (1, 256, 512, 4000, 1 << 20)), "single-token steps"
        assert not any(_in_runs(rows, 1, *heads) for rows in (1, 8, 256, 500)), "short prompts"
        assert all(_in_runs(rows, n, *heads) for rows, n in ((4096, 1), (4096, 1024), (8192, 61)))
    assert not _in_runs(4096, 1, 8, 4, kd=257) and not _in_runs(4096, 1, 8, 4, taps=3)


def _chunks(lens, H=8, kd=128, cols=256):
    ctx = SimpleNamespace(max_count=max(lens), n_seqs=len(lens))
    return native.chunked_scan_scratch(torch.empty(sum(lens), 1), ctx, H, kd, cols, delta=True) is not None


def test_scans_go_in_chunks_where_most_rows_are_in_long_sequences():
    assert _chunks([300]) and _chunks([2048]) and _chunks([300] * 8) and _chunks([2048] + [1] * 30)
    assert not _chunks([255]) and not _chunks([100] * 40)
    assert not _chunks([300] + [1] * 7) and not _chunks([160] + [1] * 60) and not _chunks([2048] + [1] * 200)
    assert not _chunks([2048], kd=129) and not _chunks([4096] * 16, H=32)


def test_a_scan_goes_row_by_row_where_the_memory_of_its_chunks_cannot_be_had(monkeypatch):
    def empty(*a, **kw):
        raise torch.OutOfMemoryError("no memory is left")

    ctx, out = SimpleNamespace(max_count=2048, n_seqs=1), torch.empty(2048, 1)
    assert native.chunked_scan_scratch(out, ctx, 8, 128, 256) is not None
    monkeypatch.setattr(native.torch, "empty", empty)
    assert native.chunked_scan_scratch(out, ctx, 8, 128, 256) is None


def test_few_row_products_ask_ahead_where_that_pays():
    def ahead(N, K, resident=592, l2=126 << 20):
        return native.library().sib_skinny_linear_ahead(*map(c_int, (-(-N // 16), resident, 16, K, l2)))

    assert ahead(18432, 2304) == ahead(16384, 2048) == ahead(256000, 2304) == ahead(128000, 2048) == 592
    for N, K in ((9216, 2304), (12288, 2048), (24576, 2304), (32000, 2048), (65536, 2048), (256000, 1536),
                 (256000, 2688), (18432, 3584), (256000, 1 << 20)):
        assert ahead(N, K) == 0, (N, K)
    assert ahead(256000, 2304, l2=96 << 20) == 0 and ahead(256000, 2304, resident=0) == 0

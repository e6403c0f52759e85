"""Which form of a kernel a call takes: the rules that the library answers without a device."""

from ctypes import c_int

from strata_inference_b200.kernels import native


def _in_runs(rows, n_seqs, H, G, kd=128, taps=4):
    return bool(native.library().sib_delta_prepare_in_runs(*map(c_int, (rows, n_seqs, H, G, kd, taps))))


def test_delta_prepare_takes_runs_where_sequences_are_long_and_rows_are_many():
    for heads in ((8, 4), (16, 8), (4, 2), (16, 2)):
        assert not any(_in_runs(n, n, *heads) for n in (1, 256, 512, 4000, 1 << 20)), "single-token steps"
        assert not any(_in_runs(rows, 1, *heads) for rows in (1, 8, 256, 500)), "short prompts"
        assert all(_in_runs(rows, n, *heads) for rows, n in ((4096, 1), (4096, 1024), (8192, 61)))
    assert not _in_runs(4096, 1, 8, 4, kd=257) and not _in_runs(4096, 1, 8, 4, taps=3)

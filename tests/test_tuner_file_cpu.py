"""The tuning file's leaf column: entries of one class that differ by it alone
are kept apart, and a line without it is one of the sample-window leaf."""


def test_entries_of_one_class_differ_by_leaf(tmp_path):
    import parode_b200 as pb

    src = tmp_path / "tune.txt"
    src.write_text("GPU 0 64 8 8 20 1 5 0.25 1\nGPU 0 64 8 8 20 1 4 0.5\nGPU 0 64 8 8 20 1 6 0.75 2\n"
                   "GPU 0 64 8 8 20 1 3 0.1 7\n")
    try:
        pb.tune_clear()
        assert pb.tune_load(str(src), gpu="GPU") == 3
        out = tmp_path / "out.txt"
        assert pb.tune_save(str(out), gpu="GPU") == 3
        got = sorted((ln.split()[9], ln.split()[7]) for ln in out.read_text().split("\n") if ln)
        assert got == [("0", "4"), ("1", "5"), ("2", "6")]
    finally:
        pb.tune_clear()

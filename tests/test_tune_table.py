"""The launch-shape table's file: entries without the present kernels' version are
left out (their shapes would pin a call to a kernel that is not the best one any
more), the others survive a round trip."""
from gpu_cross_b200 import capi

OLD = "p2.v0.x1.c1.g19.d16 8 4 1 17.170000\n"
NEW = "k2.p2.v0.x1.c1.g19.d16 1 4 1 2.500000\n"


def test_entries_of_earlier_kernels_are_left_out(built_libs, tmp_path):
    lib = capi.lib()
    src, dst = tmp_path / "in.txt", tmp_path / "out.txt"
    src.write_text(OLD + NEW + OLD.replace("c1", "c40"))
    lib.xs_tune_clear()
    try:
        capi.check(lib.xs_tune_load(str(src).encode()))
        capi.check(lib.xs_tune_save(str(dst).encode()))
        assert dst.read_text() == NEW
    finally:
        lib.xs_tune_clear()

"""Which pose calls are dealt into cells, and with how much workspace (host
rules of csrc/gd_poses.cu; nothing runs)."""
from tests import native


def test_cells_only_where_int_indexes_hold(tmp_path):
    native.run(tmp_path, r"""
  using namespace gd;
  KTables T{};
  T.lna = 128;
  T.pnp = 20000;
  CHECK(pose_work_bytes(T, 2047) == 0);
  for (int n : {2048, 16384, 16385, 1000000, 1 << 30}) {
    const size_t b = pose_work_bytes(T, n);
    CHECK(b >= 12 * (size_t)n && b < 14 * (size_t)n + (2u << 20));
  }
  // the calls that the int indexes of the cell kernels do not reach run without
  for (int n : {(1 << 30) + 1, 2147332097, 2147352500, 2147483647})
    CHECK(pose_work_bytes(T, n) == 0);
""")

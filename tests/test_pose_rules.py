"""Which pose calls are dealt into cells, and with how much workspace (host
rules of csrc/gd_poses.cu; nothing runs)."""
from tests import native


def test_cells_only_where_int_indexes_hold(tmp_path):
    native.run(tmp_path, r"""
  using namespace gd;
  KTables T{};
  T.lna = 128;
  T.pnp = 20000;
  CHECK(pose_work_bytes(T, 0.9, 148, 2047) == 0);
  for (int n : {2400, 16384, 16385, 1000000, 1 << 30}) {
    const size_t b = pose_work_bytes(T, 0.9, 148, n);
    CHECK(b >= 12 * (size_t)n && b < 14 * (size_t)n + (2u << 20));
  }
  // the calls that the int indexes of the cell kernels do not reach run without
  for (int n : {(1 << 30) + 1, 2147332097, 2147352500, 2147483647})
    CHECK(pose_work_bytes(T, 0.9, 148, n) == 0);
""")


def test_cells_only_where_they_pay(tmp_path):
    native.run(tmp_path, r"""
  auto cells = [](int n, int lna, int pnp, double far_share) {
    gd::KTables T{};
    T.lna = lna;
    T.pnp = pnp;
    return gd::pose_cells_pay(T, far_share, 148, n);
  };
  // half of the SMs idle: split over them instead
  CHECK(!cells(2048, 96, 16000, 0.9) && !cells(2368, 96, 16000, 0.9));
  CHECK(cells(2369, 96, 16000, 0.9));
  // the cells' half-filled blocks would begin another wave of few
  CHECK(cells(4000, 96, 6000, 0.7) && !cells(4700, 96, 6000, 0.7));
  CHECK(cells(8600, 96, 6000, 0.7) && !cells(9400, 96, 6000, 0.7));
  // nothing far: at no size
  for (int n = 2048; n < 2000000; n += n / 7) CHECK(!cells(n, 96, 700, 0.01));
  // many waves
  CHECK(cells(131072, 48, 2000, 0.36) && cells(131072, 48, 2000, 0.21));
  CHECK(cells(100000, 20, 800, 0.12) && !cells(60000, 48, 900, 0.02));
  CHECK(cells(30011, 48, 8000, 0.79) && cells(12345, 96, 6000, 0.7) && cells(16384, 24, 1500, 0.34));
  // one wave of blocks
  CHECK(cells(4096, 24, 1500, 0.34) && !cells(4096, 24, 1500, 0.1) && !cells(2900, 48, 1000, 0.06));
  // a few points: the deal takes longer than it saves
  CHECK(!cells(20000, 8, 100, 0.9));
  // wherever the SMs are many or few, no cells on half of them
  for (int n_sm : {16, 64, 148, 264})
    for (int n = 1; n < 16 * n_sm; n += 97) {
      gd::KTables T{};
      T.lna = 96;
      T.pnp = 16000;
      CHECK(!gd::pose_cells_pay(T, 0.9, n_sm, n));
    }
""")

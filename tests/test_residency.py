"""How many protein points stay in shared memory for a whole MC launch (host
rule pick_stages): as many as before kernels that list a chunk's points took
shared memory of their own, for every ligand size, unsplit and on clusters."""
from tests import native

# ligand atoms: resident 128-point tiles of a CTA unsplit, and with 8 per unit
TILES = {8: (56, 55), 16: (55, 52), 24: (53, 49), 32: (51, 46), 40: (48, 43), 48: (47, 41),
         56: (43, 36), 64: (44, 37), 72: (41, 34), 80: (41, 32), 88: (37, 28), 96: (34, 25),
         104: (31, 20), 112: (27, 16), 120: (27, 16)}


def test_resident_points(tmp_path):
    checks = "\n".join(f"  check({lna}, {a}, {b});" for lna, (a, b) in TILES.items())
    native.run(tmp_path, checks, r"""
bool resident(int lna, int tiles, int split, bool lists) {
  gd::KTables T{};
  T.lna = lna;
  T.pnp = tiles * split * gd::TILE_PTS;
  int ns = 0, res = 0;
  gd::pick_stages(T, gd::default_tile(lna), &ns, &res, split, lists);
  return res != 0;
}
void check(int lna, int one, int eight) {
  CHECK(resident(lna, one, 1, false));
  CHECK(resident(lna, eight, 8, false));
  CHECK(!resident(lna, gd::MAX_RESIDENT_TILES + 1, 1, false));
  // lists cost some tiles, in the kernels that have them only
  CHECK(resident(lna, one - 5, 1, true) && resident(lna, eight - 6, 8, true));
}
""")

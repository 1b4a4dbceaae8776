"""What a server lane launches next (host rule of csrc/gd_common.h): new
requests keep arriving in every round, and the members still advance."""
from tests import native


def test_members_advance_under_steady_arrivals(tmp_path):
    native.run(tmp_path, r"""
  for (int arrivals = 0; arrivals < 4; ++arrivals) {  // one in that many rounds (0: none)
    bool last_init = false;
    int fresh = 1, members = 0, mc = 0, waited = 0;
    for (int round = 0; round < 100; ++round) {
      if (arrivals && round % arrivals == 0) ++fresh;
      if (!fresh && !members) continue;
      last_init = gd::lane_inits_next(fresh > 0, members > 0, last_init);
      if (last_init) {
        CHECK(fresh > 0);
        members += fresh;
        fresh = waited = 0;
      } else {
        CHECK(members > 0);
        ++mc;
        waited += fresh > 0;
        CHECK(waited <= 1);  // a new request waits for one MC launch at most
      }
    }
    CHECK(mc >= 49);
  }
  // after an initialisation whose requests have all been cancelled
  CHECK(gd::lane_inits_next(true, false, true));
  CHECK(!gd::lane_inits_next(false, true, true) && !gd::lane_inits_next(false, true, false));
""")

"""The rule that gives a structure of a population its CTAs, against measured
launches on a B200: ms with 1, 2 and 4 CTAs a structure.  The choice may not be
slower than 4 CTAs for up to two structures an SM and 1 above by more than two
runs of one launch differ (7%)."""
from __future__ import annotations

import pytest

SMS = 148
# (structures, mitr): (1, 2, 4 CTAs) for populations of 2 and 3 species of 8 to 64 atoms, and 3 of 16 to 24 and 40 to 64
MEASURED = {
    (40, 6): [(4.7, 2.7, 2.0), (20.5, 11.3, 7.6), (11.5, 6.7, 6.9), (31.6, 19.5, 13.6)],
    (40, 500): [(464.9, 246.3, 200.4), (275.5, 184.2, 102.7), (74.8, 36.9, 37.4), (417.2, 242.6, 162.5)],
    (100, 20): [(16.9, 11.1, 16.0), (51.2, 29.7, 40.5), (37.1, 26.8, 41.5), (65.1, 44.4, 47.1)],
    (100, 200): [(187.7, 123.6, 173.9), (338.5, 195.9, 132.4), (87.1, 48.5, 87.6), (372.4, 222.4, 201.7)],
    (150, 500): [(473.2, 398.2, 579.6), (441.0, 322.6, 208.8), (88.4, 62.9, 116.0), (461.4, 302.4, 326.9)],
    (200, 200): [(187.8, 196.4, 292.9), (429.2, 232.8, 286.9), (116.2, 94.5, 176.8), (395.5, 378.6, 469.2)],
    (256, 6): [(5.7, 6.2, 9.2), (27.6, 24.7, 36.1), (19.0, 16.8, 34.0), (40.9, 35.3, 42.1)],
    (256, 100): [(102.7, 114.8, 171.9), (223.3, 178.1, 243.5), (107.4, 90.2, 163.3), (317.1, 283.3, 352.9)],
    (256, 500): [(543.0, 631.5, 926.2), (504.6, 341.6, 278.8), (128.4, 102.4, 168.5), (556.7, 392.0, 497.0)],
    (296, 200): [(243.1, 293.4, 438.6), (443.3, 302.7, 420.1), (138.1, 129.2, 218.8), (498.5, 472.2, 620.0)],
    (400, 500): [(832.1, 942.3, 1442.2), (716.6, 586.6, 822.2)],
    (1000, 500): [(1982.2, 2326.1, 3622.3), (1223.0, 1326.6, 1933.4)],
}


@pytest.mark.parametrize("S,mitr", sorted(MEASURED))
def test_never_slower_than_the_simple_rule(S, mitr):
    import maise_b200

    c = maise_b200.load_library().mbk_batch_clusters(S, mitr, SMS)
    simple = 4 if S <= 2 * SMS else 1
    for t in MEASURED[(S, mitr)]:
        t = dict(zip((1, 2, 4), t))
        assert t[c] <= 1.07 * t[simple], (c, t)


def test_fits_any_device():
    import maise_b200

    lib = maise_b200.load_library()
    for sms in (1, 3, 16, 148):
        for S in (1, 7, 300):
            for mitr in (0, 1, 500):
                assert lib.mbk_batch_clusters(S, mitr, sms) in (1, 2, 4)

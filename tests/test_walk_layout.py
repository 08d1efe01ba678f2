"""Shared memory of the launches that walk the rows (host arithmetic, no GPU)."""
import ctypes as C

import pytest

from internals import internals  # noqa: F401

OPTIN = 232448  # bytes a GB300 CTA can take


@pytest.mark.parametrize("views", [1, 8, 9, 15, 21, 31, 41, 61, 96, 160, 161, 256])
def test_a_plan_fits_wherever_the_general_layout_does(internals, views):
    """The table-driven layout is taken only within the limit, with two row caches where they fit;
    a scheduled call's fits wherever the general one does."""
    general = internals.t_general_bytes
    walk, table, sched = internals.t_walk_bytes, internals.t_table_bytes_of, internals.t_sched_bytes
    aside = 0
    for staged in (0, 1) if views <= 160 else (0,):
        for bf in (0, 1):
            for n_x in range(1, 4100, 7):
                n_rs = (n_x + 3) // 4 * 4 if staged else 0
                n_sp = (n_x + 15) // 16 * 16 if bf and staged else 0
                if general(views, n_x, n_rs, n_sp) > OPTIN:
                    continue
                two, one = (table(views, n_x, n_rs, staged, n_sp, k) for k in (2, 1))
                limit = OPTIN - 1024
                want = two if two <= limit else one if one <= limit else 0
                assert walk(views, n_x, n_rs, staged, n_sp, C.c_long(limit)) == want
                assert sched(views, n_rs, staged, n_sp) <= OPTIN
                aside += want == 0
    assert (aside > 0) == (views <= 41)  # the windows that the table is left aside in

"""Contexts share pages of page-locked status words: each reports its own status, more of them than a page holds,
from several threads, and again after all of them are gone."""
import concurrent.futures

import numpy as np
import pytest

import tild
from helpers import small_diblock

pytestmark = pytest.mark.gpu


def test_more_contexts_than_a_page_of_status_words():
    s = small_diblock(2, 1)
    far, nan = s.x.copy(), s.x.copy()
    far[3, 0], nan[3, 0] = 1e4, np.nan

    def use(k):
        """None, or the status of the failed call: every fourth context gets a far or a non-finite position."""
        c = tild.Context(s)
        try:
            if k % 4 == 1:
                c.set_state(far)
            if k % 4 == 3:
                c.set_state(nan)
            c.step(3)
        except tild.TildError as e:
            return c, e.status
        return c, None

    for _ in range(2):
        with concurrent.futures.ThreadPoolExecutor(8) as pool:
            got = list(pool.map(use, range(70)))
        want = [None, tild.ERR_BAD_INPUT, None, tild.ERR_NAN]
        assert [st for _, st in got] == [want[k % 4] for k in range(70)]
        with concurrent.futures.ThreadPoolExecutor(8) as pool:
            list(pool.map(lambda g: g[0].close(), got))

"""The task list the persistent LDL^H kernel runs (ecg_ldl_task_list), where
an update far from its panels is one task for four of them: complete, in an
order that meets every wait of the kernel (so that it cannot deadlock), and
giving the factor when executed task by task, both with the updates one by
one and with those the kernel merges at run time."""
import ctypes as C

import numpy as np
import pytest

from ecg_b200 import _lib
from test_ldl_schedule import B_, D_, NB, T_, decode, run_tasks, split

MERGE = 4


def task_list(n, workers):
    lib = _lib.load()
    cnt = C.c_longlong()
    assert lib.ecg_ldl_task_list(n, workers, None, 0, C.byref(cnt)) == 0
    out = np.zeros(cnt.value, dtype=np.uint32)
    assert lib.ecg_ldl_task_list(n, workers, C.c_void_p(out.ctypes.data), cnt.value, C.byref(cnt)) == 0
    return [decode(x) for x in out]


def grouped(s, r):
    return r >= s - s % MERGE + 8


def expected_tasks(np_):
    t = set()
    for s in range(np_):
        t.add((D_, s, s, s, 0))
        t.update((T_, s, s, c, 0) for c in range(s + 1, np_))
        for r in range(s + 1, np_):
            for c in range(r, np_):
                if grouped(s, r):
                    t.add((B_, s - s % MERGE, r, c, 1))
                else:
                    t.add((B_, s, r, c, 0))
                    if split(s, r, c):
                        t.add((B_, s, r, c, 1))
    return t


def walk(lst, np_, merge):
    """The kernel's tile counts along the list: asserts that the counts each
    task waits for are there when it is taken, and returns the updates as
    (task, panels applied).  merge: an update of its own takes the following
    panels of its group whose rows are final, as the kernel does when it
    finds them."""
    cnt = np.zeros((np_, np_), dtype=int)
    halves = {}
    done = []
    for task in lst:
        ty, s, r, c, h = task
        if ty == D_:
            assert cnt[s, s] >= s, task
            cnt[s, s] = s + 1
            done.append((task, 1))
        elif ty == T_:
            assert cnt[s, s] >= s + 1 and cnt[s, c] >= s, task
            cnt[s, c] = s + 1
            done.append((task, 1))
        else:
            g = grouped(s, r)
            last = s + MERGE - 1 if g else s
            assert cnt[r, c] >= s and cnt[last, r] >= last + 1 and cnt[last, c] >= last + 1, task
            if not g and cnt[r, c] > s:
                continue  # applied already
            m = MERGE if g else 1
            if merge and not g and not split(s, r, c) and not r == c == s + 1:
                for j in range(1, MERGE):
                    own = split(s + j, r, c) or s + j == r - 1
                    if (m == j and not own and s % MERGE + j < MERGE and s + j < r and cnt[s + j, r] > s + j
                            and cnt[s + j, c] > s + j):
                        m = j + 1
            done.append((task, m))
            if split(s, r, c) and not g:
                halves[r, c] = halves.get((r, c), 0) + 1
                if halves[r, c] % 2:
                    continue
            cnt[r, c] = s + m
    assert all(cnt[r, c] == r + 1 for r in range(np_) for c in range(r, np_))
    return done


@pytest.mark.parametrize("n,workers", [(1, 1), (65, 2), (512, 3), (513, 296), (577, 1), (640, 296), (768, 8),
                                       (832, 296), (1100, 16), (4000, 294), (10000, 294), (12800, 294)])
def test_list_is_complete_and_meets_every_wait(n, workers):
    lst = task_list(n, workers)
    np_ = (n + NB - 1) // NB
    assert len(lst) == len(set(lst)) and set(lst) == expected_tasks(np_)
    walk(lst, np_, False)
    walk(lst, np_, True)
    pos = {t: i for i, t in enumerate(lst)}
    chain = [pos[D_, 0, 0, 0, 0]]
    for s in range(np_ - 1):
        chain += [pos[T_, s, s, s + 1, 0], pos[B_, s, s + 1, s + 1, 0], pos[D_, s + 1, s + 1, s + 1, 0]]
    assert chain == sorted(chain)


@pytest.mark.parametrize("merge", [False, True])
@pytest.mark.parametrize("n", [513, 576, 640, 700, 768, 832, 1090])
def test_list_executes_to_the_ldlh_factor(n, merge):
    """9 to 18 panels: the factor reproduces the matrix within the bound of
    the list without groups, and is that list's factor."""
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    M = X @ X.conj().T / n + np.diag(rng.uniform(-2.0, 2.0, n))
    np_ = (n + NB - 1) // NB
    one = []
    for (ty, s, r, c, h), m in walk(task_list(n, 16), np_, merge):
        if ty == B_ and m > 1:
            one += [(B_, s + j, r, c, 0) for j in range(m)]
        else:
            one.append((ty, s, r, c, h))
    assert len({t for t in one if t[0] == B_}) == len([t for t in one if t[0] == B_])
    U, d = run_tasks(M, one)
    R = U.conj().T @ np.diag(d) @ U
    assert np.max(np.abs(R - M)) <= 1e-10 * np.max(np.abs(M))

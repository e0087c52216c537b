"""BigFloat's linear operations at the edges of their kernels: a CTA owns 2048
words and takes its carry-in from the aggregates below it, so numbers of one
CTA, of a word more, and of many CTAs, with carries and borrows that run
through all of them, against Python integers; and the comparison that orders a
subtraction, from several threads at once."""
from __future__ import annotations

import ctypes as C
import threading
import time

import numpy as np
import pytest

from oracle.ffi import random_words

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 2047, 2048, 2049, 4096, 6149, 300_001, 2_200_003]


def _num(pic, words, sign=True):
    return pic.DeviceBigFloat.from_words(sign, 0, np.ascontiguousarray(words, dtype=np.uint32))


def _int(x):
    bf = x.to_bf()
    assert bf.words.size == 0 or bf.words[-1] != 0
    v = int.from_bytes(bf.words.astype("<u4").tobytes(), "little") << (32 * bf.exp)
    return v if bf.sign else -v


def _val(words):
    return int.from_bytes(np.ascontiguousarray(words, dtype="<u4").tobytes(), "little")


@pytest.mark.parametrize("n", SIZES)
def test_long_carries_and_borrows(pic, n):
    ones = np.full(n, 0xFFFFFFFF, dtype=np.uint32)
    power = np.zeros(n + 1, dtype=np.uint32)
    power[n] = 1
    one = pic.DeviceBigFloat.from_u32(1)
    assert _int(_num(pic, ones).add(one)) == _val(ones) + 1          # a carry through every word
    assert _int(_num(pic, power).sub(one)) == _val(power) - 1        # a borrow through every word
    assert _int(one.sub(_num(pic, power))) == 1 - _val(power)
    assert _int(_num(pic, ones).mul_u32(0xFFFFFFFF)) == _val(ones) * 0xFFFFFFFF
    mid = np.zeros(n + 1, dtype=np.uint32)                           # the borrow clears the only word
    mid[n] = 1
    low = np.zeros(n + 1, dtype=np.uint32)
    low[n], low[0] = 1, 1
    assert _int(_num(pic, low).sub(_num(pic, mid))) == 1
    assert _int(_num(pic, mid).sub(_num(pic, low))) == -1
    assert _num(pic, low).sub(_num(pic, low)).info()[2] == 0


@pytest.mark.parametrize("n", SIZES)
def test_random_sums_and_differences(pic, n):
    a, b = random_words(n, n), random_words(n + 7, n)
    a[-1] |= 1
    b[-1] = a[-1]  # equal top words: the comparison needs words further down
    x, y = _num(pic, a), _num(pic, b)
    assert _int(x.add(y)) == _val(a) + _val(b)
    assert _int(x.sub(y)) == _val(a) - _val(b)
    assert _int(y.sub(x)) == _val(b) - _val(a)
    assert _int(x.add(_num(pic, b, sign=False))) == _val(a) - _val(b)
    assert x.ucmp(y) == (_val(a) > _val(b)) - (_val(a) < _val(b))


@pytest.mark.parametrize("n", [8191, 8192, 8193, 16385, 65535, 65536, 65537])
def test_one_launch_edges(pic, n):
    """Up to 65,536 words a cluster of CTAs of 8192 words does all of an operation;
    a difference cut to a window compares the words under it as well."""
    a, b = random_words(3 * n, n), random_words(3 * n + 1, n)
    a[n // 2:] = b[n // 2:]
    x, y = _num(pic, a), _num(pic, b)
    assert _int(x.add(y)) == _val(a) + _val(b)
    assert _int(x.sub(y)) == _val(a) - _val(b)
    assert _int(x.mul_u32(0xFFFFFFFB)) == _val(a) * 0xFFFFFFFB
    ones = np.full(n, 0xFFFFFFFF, dtype=np.uint32)
    assert _int(_num(pic, ones).add(pic.DeviceBigFloat.from_u32(1))) == _val(ones) + 1
    for lo in (0, 5, n // 2 - 1):  # the window drops the words that differ: zero
        c = a.copy()
        c[lo] ^= 1
        assert _num(pic, c).sub(x, n // 2 - 4).info()[2] == 0


def test_ordered_differences_from_several_threads(pic):
    def work(seed, bad):
        a, b = random_words(seed, 5000), random_words(seed + 1, 5000)
        a[-1] = b[-1] = 9
        x, y = _num(pic, a), _num(pic, b)
        for _ in range(40):
            if _int(x.sub(y)) != _val(a) - _val(b) or _int(y.sub(x)) != _val(b) - _val(a):
                bad.append(seed)

    bad: list[int] = []
    threads = [threading.Thread(target=work, args=(100 + 2 * i, bad)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_equal_windows_of_long_numbers(pic):
    """A difference cut to a short window in which two long numbers agree is zero
    whatever lies under the window, and costs what the window holds."""
    a = random_words(5, 1 << 24)
    b = a.copy()
    b[0] ^= 1
    x, y = _num(pic, a), _num(pic, b)
    seconds = []
    for _ in range(7):
        pic.synchronize()
        t = time.perf_counter()
        d = x.sub(y, 8)
        seconds.append(time.perf_counter() - t)
        assert d.info()[2] == 0
    assert sorted(seconds)[3] < 2e-3  # 2^24 words read by one CTA: 31 ms


def test_long_ordered_differences_from_several_threads(pic):
    """Above 65,536 words a comparison and the subtraction that reads its result are
    launches of their own over shared scratch words: no other thread's comparison may
    come between them."""
    n = 70_000

    def work(seed, bad):
        a, b = random_words(seed, n), random_words(seed + 1, n)
        a[-1] = b[-1] = 9
        a[n // 2:] = b[n // 2:]
        a[n // 2], b[n // 2] = (9, 8) if seed & 2 else (8, 9)  # the larger one differs from thread to thread
        want = _val(a) - _val(b)
        x, y = _num(pic, a), _num(pic, b)
        for _ in range(40):
            if _int(x.sub(y)) != want or _int(y.sub(x)) != -want:
                bad.append(seed)

    bad: list[int] = []
    threads = [threading.Thread(target=work, args=(200 + 2 * i, bad)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


CHUNK, DIRECT, GROUP = 2048, 8192, 512  # words of a chunk; chunks scanned directly; chunks of a group


@pytest.mark.parametrize("n", [DIRECT * CHUNK, DIRECT * CHUNK + 1, 20_000_003])
def test_carries_through_groups_of_chunks(pic, n):
    """More than 8192 chunks: a carry through all of them, through some of them up to
    or from the edge of a chunk and of a group, and a borrow the same way."""
    one = pic.DeviceBigFloat.from_u32(1)
    ones = np.full(n, 0xFFFFFFFF, dtype=np.uint32)
    got = _num(pic, ones).add(one).to_bf()
    assert got.words.size == n + 1 and got.words[n] == 1 and not got.words[:n].any()
    got = got.words
    got = _num(pic, got).sub(one).to_bf()
    assert got.words.size == n and np.all(got.words == 0xFFFFFFFF)
    got = _num(pic, ones).mul_u32(0xFFFFFFFF).to_bf().words  # (B^n - 1)(B - 1)
    assert got[0] == 1 and np.all(got[1:n] == 0xFFFFFFFF) and got[n] == 0xFFFFFFFE
    for c in (1, GROUP, GROUP + 1, 3 * GROUP - 1, DIRECT - 1):
        for q in (c * CHUNK - 1, c * CHUNK):
            w = ones.copy()
            w[q] = 7
            got = _num(pic, w).add(one).to_bf().words  # stops at q
            assert not got[:q].any() and got[q] == 8 and np.all(got[q + 1:] == 0xFFFFFFFF)
            w = np.zeros(n, dtype=np.uint32)
            w[q], w[n - 1] = 7, 5
            low = np.zeros(2 * CHUNK + 1, dtype=np.uint32)
            low[0], low[-1] = 1, 1
            if q > 2 * CHUNK:  # two borrows, the second from a chunk further up
                got = _num(pic, w).sub(_num(pic, low)).to_bf().words
                assert np.all(got[:2 * CHUNK] == 0xFFFFFFFF) and got[2 * CHUNK] == 0xFFFFFFFE
                assert np.all(got[2 * CHUNK + 1:q] == 0xFFFFFFFF) and got[q] == 6 and got[n - 1] == 5


def test_long_runs_cost_what_their_words_cost(pic, torch_cuda):
    """The carries through a run of all-ones or zero words take time in proportion."""
    torch = torch_cuda
    n = 400_000_000

    def number(t):
        out = C.c_void_p()
        torch.cuda.synchronize()
        pic.check(pic.lib().pic_bf_from_device(C.byref(out), 1, 0, t.data_ptr(), n, None))
        return pic.DeviceBigFloat(out.value)

    def cost(x, y):
        seconds = []
        for _ in range(5):
            pic.synchronize()
            t = time.perf_counter()
            z = x.sub(y)
            pic.synchronize()
            seconds.append(time.perf_counter() - t)
            del z
        return sorted(seconds)[2]

    ones = number(torch.full((n,), -1, dtype=torch.int32, device="cuda"))
    a = torch.randint(1, 1 << 31, (n,), dtype=torch.int32, device="cuda")
    x, y = number(a), number(a ^ 0x5555)
    assert cost(ones, ones) < 3 * cost(x, y)  # 7 times before groups

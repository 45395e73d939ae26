"""How messages that are given as tiles reach the native library, on the CPU: a stand-in for its entry points that keeps what each call hands
over, and the oracle's library, which has no entry point for tiles."""
import ctypes as C
import importlib

import numpy as np
import pytest

SLOTS = 64


class Recorder:
    """Entry points encrypt_tiles and encrypt_many of a library, as the messages [count][SLOTS] that the call would encrypt."""

    def __init__(self, capi):
        self.lib = capi.Lib.__new__(capi.Lib)
        self.lib.slots, self.lib.L, self.lib.ctx = SLOTS, 3, None
        self.lib.has = lambda name: True
        self.lib._fn = lambda name: getattr(self, name, lambda *a: 0)
        self.called = self.messages = None

    @staticmethod
    def _row(parts):
        m = np.zeros(SLOTS)
        flat = np.concatenate(parts, axis=1).reshape(-1)
        m[:flat.size] = flat
        return m

    def encrypt_tiles(self, ctx, ptr, across, rows, cols, count, level, nonces, out):
        across, rows, cols = across.value, rows.value, cols.value
        tile = lambda p: np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_double)), (rows, cols)).copy()
        self.called = "encrypt_tiles"
        self.messages = np.stack([self._row([tile(ptr[i * across + t]) for t in range(across)]) for i in range(count.value)])
        return 0

    def encrypt_many(self, ctx, re, im, n, count, level, nonces, out):
        self.called = "encrypt_many"
        self.messages = np.ctypeslib.as_array(C.cast(re, C.POINTER(C.c_double)), (count.value, n.value)).copy()
        return 0


@pytest.fixture
def rec(pkg):
    return Recorder(importlib.import_module(pkg.__name__ + ".capi"))


@pytest.mark.parametrize("groups", [(2, 2), (2, 1, 3), (1, 2), (2, 1), (3, 1, 2)])
def test_every_message_keeps_its_own_tiles(rec, groups):
    """Groups of as many tiles each go to the tile entry point, uneven ones are laid out: two tiles, one, three."""
    rng = np.random.default_rng(len(groups))
    tiles = [[rng.uniform(-1, 1, (3, 4)) for _ in range(n)] for n in groups]
    rec.lib.encrypt_tiles(tiles, 2, range(len(groups)))
    assert np.array_equal(rec.messages, np.stack([Recorder._row(g) for g in tiles]))
    assert rec.called == ("encrypt_tiles" if len(set(groups)) == 1 else "encrypt_many")


def test_tiles_of_other_forms_are_laid_out(rec):
    """Tiles of unequal width, and stacks of matrices, whose second axis they are joined on."""
    a, b, c = np.ones((4, 3)), np.full((4, 5), 2.0), np.arange(24.0).reshape(2, 3, 4)
    rec.lib.encrypt_tiles([[a, b]], 2, [1])
    assert np.array_equal(rec.messages, Recorder._row([a, b])[None])
    rec.lib.encrypt_tiles([[c, -c]], 2, [1])
    assert np.array_equal(rec.messages, Recorder._row([c, -c])[None])
    for bad in ([[]], [[a], []], [[np.ones(4)]], [[a, np.ones((3, 3))]], [[np.ones((8, 5)), np.ones((8, 4))]]):
        with pytest.raises((ValueError, IndexError)):
            rec.lib.encrypt_tiles(bad, 2, range(len(bad)))


def test_encrypt2_many_takes_pairs_only(pkg, rec):
    """Lists, tuples, arrays and iterators of two tiles; three or one are refused before anything is encrypted."""
    hemmer = importlib.import_module(pkg.__name__ + ".hemmer")
    H = hemmer.Hemmer.__new__(hemmer.Hemmer)
    H.lib = rec.lib
    rng = np.random.default_rng(4)
    a = [rng.uniform(-1, 1, (3, 4)) for _ in range(6)]
    got = H.encrypt2_many([(a[0], a[1]), [a[2], a[3]], iter((a[4], a[5]))], [1, 2, 3])
    assert got.shape == (3, 4, 8)
    assert np.array_equal(rec.messages, np.stack([Recorder._row([a[k], a[k + 1]]) for k in (0, 2, 4)]))
    H.encrypt2_many(np.stack(a[:2])[None], [1])
    assert np.array_equal(rec.messages, Recorder._row(a[:2])[None])
    rec.called = None
    for bad in ([a[:3]], [a[:1]], [a[:2], a[:3]], [a[:2], a[2:3], a[3:6]]):
        with pytest.raises(ValueError):
            H.encrypt2_many(bad, range(len(bad)))
    assert rec.called is None


def test_one_nonce_a_message(rec, orc_small):
    """Missing nonces were zeros: messages under one nonce share their randomness, and the difference of the ciphertexts gives that of the messages."""
    msgs = np.random.default_rng(5).uniform(-1, 1, (3, 16))
    tiles = [[m.reshape(4, 4)] for m in msgs]
    for lib in (rec.lib, orc_small):
        for nonces in ([], [7, 8], [7, 8, 9, 10], range(2)):
            with pytest.raises(ValueError):
                lib.encrypt_many(msgs, 2, nonces)
            with pytest.raises(ValueError):
                lib.encrypt_tiles(tiles, 2, nonces)
    assert rec.called is None
    want = [orc_small.ct_export(orc_small.encrypt(orc_small.encode(m, 2), k)) for m, k in zip(msgs, (7, 8, 9))]
    for got in (orc_small.encrypt_many(msgs, 2, iter((7, 8, 9))), orc_small.encrypt_tiles(tiles, 2, np.arange(7, 10))):
        assert np.array_equal(orc_small.ct_export(got), np.concatenate(want))

"""Encoding, sampling, encryption and decryption on the device against the oracle, whose embedding, error polynomials and CRT lift are
host code with the same sequence of IEEE operations: residues and decoded values are compared bit for bit.  Messages go up in
chunks of four and values come down in chunks of eight, through two buffers each, so batches lie on both sides of one to five chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(request, size):
    return request.getfixturevalue(f"gpu_{size}"), request.getfixturevalue(f"orc_{size}")


def _messages(rng, count, slots, cplx):
    z = rng.uniform(-1, 1, (count, slots))
    return z + 1j * rng.uniform(-1, 1, (count, slots)) if cplx else z


@pytest.mark.parametrize("size,level,count,slots,cplx", [
    ("small", 0, 1, 1, False), ("small", 8, 9, 511, True), ("mid", 3, 17, 2048, True), ("mid", 1, 8, 0, False),
    ("full", 12, 9, 32768, False), ("full", 0, 2, 32767, True), ("full", 1, 17, 129, True), ("full", 4, 8, 20000, False)])
def test_encrypt_and_decrypt_equal_the_oracle(request, size, level, count, slots, cplx):
    g, o = _pair(request, size)
    msgs = _messages(np.random.default_rng(level * 100 + count), count, slots, cplx)
    nonces = [2**63 + 5 * k for k in range(count)]
    ct = g.encrypt_many(msgs, level, nonces)
    got = g.ct_export(ct)
    values = g.decrypt_many([(ct, k) for k in reversed(range(count))])[::-1]
    for k in sorted({0, min(7, count - 1), min(8, count - 1), count - 1}):
        ref = o.encrypt(o.encode(msgs[k], level), nonces[k])
        assert np.array_equal(got[k:k + 1], o.ct_export(ref)), f"ciphertext {k}"
        assert np.array_equal(values[k], o.decrypt(ref)), f"values {k}"
        assert np.array_equal(values[k], g.decrypt(ct, k))


@pytest.mark.parametrize("size", ["small", "full"])
@pytest.mark.parametrize("scale", [1e-300, 2.0**-20, 2.0**20, 1e30])
def test_rounding_at_the_ends_of_the_range(request, size, scale):
    """Coefficients that vanish, that leave the 51 bits of the short reduction, and that do not fit 64 bits (which saturate as on the host)."""
    g, o = _pair(request, size)
    z = _messages(np.random.default_rng(3), 1, g.slots, True)[0] * scale
    z[1] = -0.0
    for level in (1, g.L):
        assert np.array_equal(g.pt_export(g.encode(z, level)), o.pt_export(o.encode(z, level)))
        p, q = g.encode(z, level), o.encode(z, level)
        assert np.array_equal(g.decode(p), o.decode(q))


def test_not_a_number_and_infinity_encode_as_on_the_host(gpu_small, orc_small):
    z = np.zeros(gpu_small.slots)
    for bad in (np.nan, np.inf, -np.inf):
        z[3] = bad
        assert np.array_equal(gpu_small.pt_export(gpu_small.encode(z, 2)), orc_small.pt_export(orc_small.encode(z, 2)))


@pytest.mark.parametrize("size", ["small", "full"])
def test_decoding_of_uniform_residues(request, size):
    """Every value of the lift is met: both halves of q_0 and of q_0 q_1, one to three polynomials, one and two factors of the scale."""
    from conftest import rand_ct_residues
    g, o = _pair(request, size)
    for level, polys, power in ((0, 2, 1), (1, 3, 2), (3, 2, 2)):
        data = rand_ct_residues(g, level, polys, 1, seed=level + 7)
        cts = []
        for lib in (g, o):
            ct = lib.ct_create(level, polys, 1, power)
            lib.ct_import(ct, data)
            cts.append(ct)
        assert np.array_equal(g.decrypt(cts[0]), o.decrypt(cts[1])), (level, polys, power)


@pytest.mark.parametrize("size", ["small", "full"])
def test_members_with_one_limb_among_others(request, size):
    """Chunks of eight whose members have one limb each, some two, one polynomial or three."""
    g, o = _pair(request, size)
    from conftest import rand_ct_residues
    cts = []
    for lib in (g, o):
        cts.append([])
        for k, (level, polys) in enumerate([(0, 2), (3, 2), (0, 3), (1, 2)]):
            ct = lib.ct_create(level, polys, 1)
            lib.ct_import(ct, rand_ct_residues(g, level, polys, 1, seed=30 + k))
            cts[-1].append(ct)
    want = [o.decrypt(ct) for ct in cts[1]]
    order = [0, 2] * 4 + [0, 1, 2, 3] * 2 + [0, 3, 2]
    got = g.decrypt_many([(cts[0][k], 0) for k in order])
    for row, k in zip(got, order):
        assert np.array_equal(row, want[k])


@pytest.mark.parametrize("size", ["small", "full"])
def test_switching_keys_equal_the_oracle(request, size):
    g, o = _pair(request, size)
    for galois in (0, g.galois(3)):
        g.gen_rot_keys([3]); o.gen_rot_keys([3])
        assert np.array_equal(g.evk_export(galois), o.evk_export(galois))


@pytest.mark.parametrize("size,count,across,rows,cols", [("small", 1, 1, 1, 1), ("mid", 9, 2, 8, 4), ("full", 17, 2, 128, 128), ("full", 3, 3, 5, 7), ("full", 8, 1, 181, 181)])
def test_tiles_side_by_side_equal_their_messages(request, size, count, across, rows, cols):
    g = request.getfixturevalue(f"gpu_{size}")
    rng = np.random.default_rng(count)
    tiles = [[rng.uniform(-1, 1, (rows, cols)) for _ in range(across)] for _ in range(count)]
    tiles[0][0] = np.asfortranarray(tiles[0][0])  # not in row-major order: copied first
    msgs = np.stack([np.concatenate(t, axis=1).reshape(-1) for t in tiles])
    nonces = list(range(50, 50 + count))
    assert np.array_equal(g.ct_export(g.encrypt_tiles(tiles, 2, nonces)), g.ct_export(g.encrypt_many(msgs, 2, nonces)))


def test_tiles_that_are_refused_or_take_the_general_path(pkg, gpu_small):
    g = gpu_small
    wide = np.ones((2, g.slots // 2 + 1))
    for bad in ([[wide]], [[wide, wide]]):
        with pytest.raises((pkg.HBError, ValueError)):
            g.encrypt_tiles(bad, 2, [1])
    a, b = np.ones((4, 3)), np.ones((4, 5))
    assert np.array_equal(g.ct_export(g.encrypt_tiles([[a, b]], 2, [9])), g.ct_export(g.encrypt_many(np.ones((1, 32)), 2, [9])))
    assert np.array_equal(g.ct_export(g.encrypt_tiles([[np.zeros((0, 4))]], 2, [9])), g.ct_export(g.encrypt_many(np.zeros((1, 4)), 2, [9])))
    rng = np.random.default_rng(6)
    uneven = [[rng.uniform(-1, 1, (8, 8)) for _ in range(k)] for k in (2, 1, 3)]  # as many tiles as three messages of two
    msgs = np.zeros((3, g.slots))
    for m, t in zip(msgs, uneven):
        m[:64 * len(t)] = np.concatenate(t, axis=1).reshape(-1)
    assert np.array_equal(g.ct_export(g.encrypt_tiles(uneven, 2, [4, 5, 6])), g.ct_export(g.encrypt_many(msgs, 2, [4, 5, 6])))


@pytest.mark.parametrize("count", [4, 16, 17, 33])
def test_members_drawn_ahead_equal_single_encryptions(gpu_full, count):
    """Uniform parts and errors are drawn for up to sixteen members before their messages; messages that saturate and that vanish among them."""
    g = gpu_full
    msgs = _messages(np.random.default_rng(count), count, g.slots, True)
    msgs[0] *= 1e30
    msgs[-1] *= 1e-300
    nonces = [2**64 - 1 - 3 * k for k in range(count)]
    got = g.ct_export(g.encrypt_many(msgs, 2, nonces))
    for k in range(count):
        assert np.array_equal(got[k:k + 1], g.ct_export(g.encrypt(g.encode(msgs[k], 2), nonces[k]))), f"member {k}"


@pytest.mark.parametrize("sigma", [9.7, 9.8])
def test_errors_on_either_side_of_a_byte(pkg, sigma):
    """A table of 127 magnitudes is drawn ahead into bytes, one of 128 is not."""
    g = pkg.open_gpu(pkg.make_params(log_n=16, max_level=2, dnum=2, num_special=2, hamming_weight=64, sigma=sigma))
    g.keygen()
    msgs = _messages(np.random.default_rng(1), 2, g.slots, False)
    got = g.ct_export(g.encrypt_many(msgs, 1, [5, 6]))
    for k in range(2):
        assert np.array_equal(got[k:k + 1], g.ct_export(g.encrypt(g.encode(msgs[k], 1), 5 + k))), f"member {k}"
    g.close()


def test_a_cap_of_one_thread_starts_no_other(gpu_full):
    """set_host_threads caps all threads of a call: with one, the caller alone asks for pages and copies the values."""
    import os
    import threading

    from conftest import rand_ct_residues
    g = gpu_full
    level, batch = 1, 16
    x = g.ct_create(level, 2, batch)
    g.ct_import(x, rand_ct_residues(g, level, 2, batch, seed=3))
    items = [(x, k) for k in range(batch)]
    counts, stop = [], threading.Event()

    def watch():
        while not stop.is_set():
            counts.append(len(os.listdir("/proc/self/task")))

    g.set_host_threads(1)
    try:
        keep = [g.decrypt_many(items)]
        watcher = threading.Thread(target=watch)
        watcher.start()
        while len(counts) < 20:
            pass
        before = max(counts[:20])
        keep += [g.decrypt_many(items) for _ in range(40)]
        stop.set()
        watcher.join()
    finally:
        g.set_host_threads(0)
    assert max(counts) == before
    assert all(np.array_equal(keep[0], z) for z in keep)

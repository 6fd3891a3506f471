"""The window FFT's exchanges (pypty_gb300/csrc/window_fft.cuh) restated on the CPU: what its two
block barriers per transform pair rely on, and its bank conflicts.

A warp's 32 x 32 transpose and its stores of the cross-warp exchange stay inside the warp's own
8 KB part of the buffer; a thread's stores in the inverse's round 3 go to the words it loaded in
the forward's round 3; every 16-byte word that is loaded has been stored once, by the thread that
holds that element; every quarter-warp of 16-byte accesses touches 8 distinct bank quads and every
warp of 4-byte accesses 32 distinct banks."""
import numpy as np
import pytest


def geo(W):
    A = W // 32
    C, T = 32 // A, W * W // 32
    Bq = W // C
    return A, C, Bq, 32 // Bq, T // C, T


def transpose_word(k, row):            # float index of (k1 = k, local row) in a plane of the warp's part
    return k * 32 + ((((row >> 2) ^ (k & 7)) << 2) | (row & 3))


def quads(words, lanes=8):             # 16-byte words of a warp -> distinct bank quads per quarter-warp
    return [len({w % 8 for w in words[i:i + lanes]}) for i in range(0, 32, lanes)]


@pytest.mark.parametrize("W", [64, 128])
def test_transpose_inside_a_warp(W):
    A, C, Bq, Q, S3, T = geo(W)
    seen = set()
    for k in range(32):                # round 1 stores: lane = local row, 4 bytes
        words = [transpose_word(k, row) for row in range(32)]
        assert len({w % 32 for w in words}) == 32
        seen.update(words)
    assert seen == set(range(1024))
    for c in range(8):                 # round 2 loads: lane = k1, one 16-byte word = local rows 4c .. 4c+3
        words = [lane * 8 + (c ^ (lane & 7)) for lane in range(32)]
        assert quads(words) == [8] * 4
        for lane, w in enumerate(words):
            assert [4 * w + r for r in range(4)] == [transpose_word(lane, 4 * c + r) for r in range(4)]
    # local row r of warp m2 is image row Bq*(r // A) + m2 and x residue r % A
    rows = {(Bq * (r // A) + m2, r % A) for m2 in range(Bq) for r in range(32)}
    assert rows == {(y, n2) for y in range(W) for n2 in range(A)}


@pytest.mark.parametrize("W", [64, 128])
def test_cross_warp_exchange(W):
    A, C, Bq, Q, S3, T = geo(W)
    H, stored = W // 2, {}
    for m2 in range(Bq):               # round 2 stores, word (kx, kx + W/2) of row m2*C + j1
        for j1 in range(C):
            for half in range(1 if A == 2 else 2):
                words = [(m2 * C + j1) * H + lane + 32 * half for lane in range(32)]
                assert quads(words) == [8] * 4
                for lane, w in enumerate(words):
                    assert m2 * 512 <= w < (m2 + 1) * 512      # the warp's own part
                    assert w not in stored
                    stored[w] = (m2, j1, lane + 32 * half)
    assert len(stored) == W * H
    loaded = set()
    for warp in range(T // 32):        # round 3 loads; the inverse stores to the same words
        for q in range(Q // 2):
            for r in range(Bq):
                words = []
                for lane in range(32):
                    t = warp * 32 + lane
                    g, j1 = t % S3, t // S3
                    w = j1 * H + g + r * C * H + S3 * q
                    assert stored[w] == (r, j1, g + S3 * q) and w not in loaded
                    loaded.add(w)
                    words.append(w)
                assert quads(words) == [8] * 4
    assert len(loaded) == len(stored)
    # the pack's frequencies, as the element-wise code addresses them
    freq = {(t // S3 + C * ((i >> 1) % Bq), t % S3 + S3 * ((i >> 1) // Bq) + (W // 2) * (i & 1))
            for t in range(T) for i in range(32)}
    assert len(freq) == W * W == len(np.unique([ky * W + kx for ky, kx in freq]))

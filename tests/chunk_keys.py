"""Keys that crowd in the wizard's chunk dictionary: its hash restated and inverted, so that a test can choose where
its keys are placed."""
import numpy as np

M = 0xFFFFFFFF
MUL = (0x9E3779B1, 0x85EBCA77, 0xC2B2AE3D)


def _f(x, mul, shift):
    f = (x.astype(np.uint64) * np.uint64(mul)) & np.uint64(M)
    return f ^ (f >> np.uint64(shift))


def hash64(x):
    x = np.asarray(x, np.uint64)
    lo, hi = x & np.uint64(M), x >> np.uint64(32)
    hi = (hi + _f(lo, MUL[0], 15)) & np.uint64(M)
    lo = (lo + _f(hi, MUL[1], 13)) & np.uint64(M)
    hi = (hi + _f(lo, MUL[2], 16)) & np.uint64(M)
    return hi.astype(np.uint32), lo.astype(np.uint32)


def key64(place, other):
    """The 64-bit key of a hash."""
    hi, lo = np.broadcast_arrays(np.atleast_1d(np.asarray(place, np.uint64)), np.asarray(other, np.uint64))
    hi = (hi - _f(lo, MUL[2], 16)) & np.uint64(M)
    lo = (lo - _f(hi, MUL[1], 13)) & np.uint64(M)
    hi = (hi - _f(lo, MUL[0], 15)) & np.uint64(M)
    return (hi << np.uint64(32)) | lo


def key32(place):
    """The 32-bit key of a place: the finaliser of MurmurHash3 backwards."""
    x = np.asarray(place, np.uint64)
    x = x ^ (x >> np.uint64(16))
    x = (x * np.uint64(pow(0xC2B2AE35, -1, 1 << 32))) & np.uint64(M)
    x = x ^ (x >> np.uint64(13)) ^ (x >> np.uint64(26))
    x = (x * np.uint64(pow(0x85EBCA6B, -1, 1 << 32))) & np.uint64(M)
    x = x ^ (x >> np.uint64(16))
    return x.astype(np.uint32)

"""Partial sums of the sums at targets: whatever room a context has from earlier target counts, the
segments of a launch fit it, cover every source and are no more than the count asks for (the C++ host
functions, called by their mangled names)."""
import ctypes

from ves3d_b200 import _lib

TILE = 256  # sources per tile of the kernel


def test_segments_fit_their_room():
    L = ctypes.CDLL(_lib.LIB_PATH)
    doubles = L._ZN5ves3d20targets_part_doublesEl
    doubles.restype, doubles.argtypes = ctypes.c_size_t, [ctypes.c_long]
    segments = L._ZN5ves3d16targets_segmentsEllmPl
    segments.restype = ctypes.c_long
    segments.argtypes = [ctypes.c_long, ctypes.c_long, ctypes.c_size_t, ctypes.POINTER(ctypes.c_long)]
    counts = sorted({1, 50, 63, 64, 65, 4736, 4737, 9472, 9473, 20000, 37888, 60000, 75776, 75777, 200000} |
                    {int(1.07 ** k) for k in range(1, 180)})
    rooms = sorted({0} | {doubles(m) for m in counts})
    assert doubles(9472) > doubles(20000) > 0  # why the room is not a function of the count's maximum
    per = ctypes.c_long()
    for m in counts:
        for room in rooms:
            for n in (1, 255, 257, 8191, 32400, 700000):
                s = segments(n, m, room, ctypes.byref(per))
                tiles = -(-n // TILE)
                assert s >= 1 and (s == 1 or 3 * m * s <= room)
                assert (s - 1) * per.value < tiles <= s * per.value
                if room >= doubles(m):
                    assert s == segments(n, m, doubles(m), None)

"""CPU restatement of the addressing of the FP64 H.X kernel's tiles in shared
memory: every point that an output reads was copied, to its own place inside
the box, for every lattice size."""
import pytest

THREADS, ITERS, SMEM = 256, 5, 113 * 1024


def _tiling(n):
    best = None
    for tx in range(1, min(n, 16) + 1):
        for ty in range(1, min(n, 16) + 1):
            for tz in range(1, min(n, 16) + 1):
                pts = tx * ty * tz
                if pts > THREADS:
                    continue
                thr = (pts + 31) // 32 * 32
                px = tx + 8 if tx % 8 else tx + 4
                pz = px * (ty + 4) + (4 if px % 2 else 0)
                P = tx + px * (ty - 1) + pz * (tz + 3)
                points = pts + 4 * (ty * tz + tx * tz + tx * ty)
                iters = (points + thr - 1) // thr
                if iters > ITERS or P * 68 + 72 * thr > SMEM:
                    continue
                tiles = 1
                for t in (tx, ty, tz):
                    tiles *= (n + t - 1) // t
                cost = tiles * thr * (4.4 + iters)
                if best is None or cost < best[0]:
                    best = cost, tx, ty, tz, px, pz, P, points
    return best[1:]


@pytest.mark.parametrize("n", [2, 3, 4, 5, 7, 9, 12, 15, 16, 17, 23, 30, 31,
                               36, 40, 47, 48, 64, 81])
def test_box_holds_every_stencil(n):
    tx, ty, tz, px, pz, P, points = _tiling(n)

    def layer(h, t):
        return h - 2 if h < 2 else t + h - 2

    at = {}
    pts, hx, hy = tx * ty * tz, 4 * ty * tz, 4 * tx * tz
    for q in range(points):
        b = q
        if b < pts:
            p = b % tx, b // tx % ty, b // (tx * ty)
        elif b < pts + hx:
            b -= pts
            p = layer(b & 3, tx), (b >> 2) % ty, (b >> 2) // ty
        elif b < pts + hx + hy:
            b -= pts + hx
            p = b % tx, layer(b // tx & 3, ty), b // (4 * tx)
        else:
            b -= pts + hx + hy
            p = b % tx, b // tx % ty, layer(b // (tx * ty), tz)
        a = p[0] + px * p[1] + pz * (p[2] + 2)
        assert 0 <= a < P and a not in at
        at[a] = p
    for q in range(pts):
        i, j, k = q % tx, q // tx % ty, q // (tx * ty)
        base = i + px * j + pz * (k + 2)
        for m in (-2, -1, 1, 2):
            assert at[base + m] == (i + m, j, k)
            assert at[base + m * px] == (i, j + m, k)
            assert at[base + m * pz] == (i, j, k + m)

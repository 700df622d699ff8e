"""The split and the messages of k_resident, restated on the CPU: every value a tile waits for is the
neighbouring cell the stencil needs, sent in the pass before, from one slot per cell and colour that
nobody overwrites before it is read; every index stays inside its buffer."""
import pytest

BOX = 72


def plan(NX, NY, NZ, sms=148):
    """resident_plan: (R, pairs of planes per warp, tiles along positions, tiles along rows) or None; without its
    rule on how full the tiles must be beyond 30 planes."""
    HN = (NX + 3) // 2
    nxb = (HN + 31) // 32
    np_ = 1 if NZ <= 30 else 2
    if NZ > 60:
        return None
    for R in range(1, (8 if np_ == 1 else 4) + 1):
        ntj = -(-NY // R)
        if nxb * ntj <= sms:
            return R, np_, nxb, ntj
    return None


def b_shared(R, np_):
    return R <= (5 if np_ == 1 else 2)


def cell(p, j, k, c):
    """(i, j, k) of position p of colour c's half-row (j, k)."""
    return 2 * p + ((1 + c + j + k) & 1), j, k


@pytest.mark.parametrize("n", [(40, 40, 3), (41, 37, 4), (130, 9, 2), (63, 62, 3), (62, 63, 3), (200, 150, 2), (64, 1, 5),
                               (121, 117, 33)])
def test_messages_are_the_neighbours(n):
    NX, NY, NZ = n
    R, _, nxb, ntj = plan(NX, NY, NZ)
    HN = (NX + 3) // 2
    tiles = nxb * ntj
    assert tiles <= 148 and nxb * 32 >= HN and ntj * R >= NY
    box = {}
    NZe = (NZ + 1) & ~1
    size = tiles * NZe * 2 * BOX

    def slot(t, pl, c, s):
        a = ((t * NZe + pl) * 2 + c) * BOX + s
        assert 0 <= s < BOX and 0 <= a < size
        return a

    def send(n_pass, c):
        for t in range(tiles):
            xb, tj = t % nxb, t // nxb
            for pl in range(NZ):
                k = pl + 1
                for r in range(R):
                    j = 1 + tj * R + r
                    e = (1 + c + j + k) & 1
                    if r == 0 and tj > 0:
                        for lane in range(32):
                            box[slot(t, pl, c, lane)] = (n_pass, cell(xb * 32 + lane, j, k, c))
                    if r == R - 1 and tj + 1 < ntj:
                        for lane in range(32):
                            box[slot(t, pl, c, 32 + lane)] = (n_pass, cell(xb * 32 + lane, j, k, c))
                    if e and xb + 1 < nxb:
                        box[slot(t, pl, c, 64 + r)] = (n_pass, cell(xb * 32 + 31, j, k, c))
                    if not e and xb > 0:
                        box[slot(t, pl, c, 64 + r)] = (n_pass, cell(xb * 32, j, k, c))

    def read(n_pass, c):
        """Messages of colour c made in pass n_pass, read by the update of colour 1 - c."""
        used = 0
        for t in range(tiles):
            xb, tj = t % nxb, t // nxb
            j0 = 1 + tj * R
            for pl in range(NZ):
                k = pl + 1
                for lane in range(32):
                    p = xb * 32 + lane
                    for on, tt, s, j in ((tj > 0, t - nxb, 32 + lane, j0 - 1), (tj + 1 < ntj, t + nxb, lane, j0 + R)):
                        if not on:
                            # the row beyond is outside the interior (or has no cells at all)
                            assert j == 0 or j > NY
                            continue
                        own = cell(p, j0 if j < j0 else j0 + R - 1, k, 1 - c)
                        assert box[slot(tt, pl, c, s)] == (n_pass, (own[0], j, k))
                        used += 1
                for r in range(R):
                    j = j0 + r
                    e = (1 + (1 - c) + j + k) & 1  # the updated cell's
                    lane, on, tt = (31, xb + 1 < nxb, t + 1) if e else (0, xb > 0, t - 1)
                    i = cell(xb * 32 + lane, j, k, 1 - c)[0]
                    if on:
                        assert box[slot(tt, pl, c, 64 + r)] == (n_pass, (i + (1 if e else -1), j, k))
                        used += 1
        return used

    total = 0
    send(0, 0)
    for n_pass in range(1, 10):
        c = n_pass & 1
        total += read(n_pass - 1, 1 - c)
        send(n_pass, c)
    total += read(8, 0) + read(9, 1)  # CalcAX behind the last pass
    assert total > 0 or tiles == 1


@pytest.mark.parametrize("NZ", [1, 9, 29, 30, 31, 59, 60, 61])
def test_split_covers_and_fits(NZ):
    """Every grid with a split has a tile per SM at most, rows within the kernel's limits and shared
    memory within a block's; x and b indices stay inside their arrays."""
    seen = 0
    for NX in (1, 2, 40, 61, 62, 63, 121, 181, 240, 254, 255, 300, 480):
        for NY in (1, 7, 8, 40, 117, 179, 240, 259, 260, 300):
            pl = plan(NX, NY, NZ)
            if pl is None:
                continue
            seen += 1
            R, np_, nxb, ntj = pl
            assert (ntj - 1) * R < NY <= ntj * R
            warps = -(-NZ // (2 * np_))
            assert warps <= 15 and warps * np_ * 2 >= NZ
            x_elems = ((NZ + 1) // 2 * 2 + 2) * 2 * R * 34
            # the lane's elements read by the first and the last pair: the planes of zeros around them
            pl = 2 * R * 34
            assert pl + 0 - pl >= 0
            assert pl + ((NZ + 1) // 2 * 2 - 2 + 2) * pl + R * 34 + (R - 1) * 34 + 1 + 32 == x_elems - 1
            pairs = (NZ + 1) // 2
            own = pairs * 2 * R * 32 * (4 + (16 if b_shared(R, np_) else 0))  # classes and b
            # room for 500 classes at least beside them
            assert 8 * (x_elems + 8 * 500) + own + 512 <= 232448
    assert seen or NZ > 60
    if NZ == 30:
        assert plan(240, 240, 30) == (7, 1, 4, 35) and plan(254, 259, 30) == (7, 1, 4, 37)
        assert plan(254, 296, 30) == (8, 1, 4, 37)
        assert plan(120, 120, 30)[0] == 2 and plan(40, 40, 30)[0] == 1 and plan(300, 300, 30) is None


@pytest.mark.parametrize("NY", [1, 7, 8, 9, 40, 117, 240, 259])
@pytest.mark.parametrize("R", range(1, 9))
def test_row_sums_have_one_owner(NY, R):
    """Every row of a group of 8 is posted by one tile, and one tile adds each group."""
    ntj = -(-NY // R)
    owners = {}
    for tj in range(ntj):
        group = (tj * R + 7) >> 3
        if group * 8 < tj * R + R and group * 8 < NY:
            owners.setdefault(group, []).append(tj)
    assert sorted(owners) == list(range(-(-NY // 8))) and all(len(v) == 1 for v in owners.values())


LAYOUT = r"""
#include <cstdio>
#include "h2g_resident.cuh"
using namespace h2g;
int main() {
  printf("%d %d %d %d %d\n", kRsRowPitch, kRsBox, kRsTabRow, kRsMaxTab, kRsMaxWarps);
  for (int R = 1; R <= kRsMaxRows; ++R)
    for (int NZ = 1; NZ <= 4 * kRsMaxWarps; ++NZ)
      for (int bs = 0; bs < 2; ++bs)
        printf("%d %d %d %zu %zu\n", R, NZ, bs, rs_x_elems(R, NZ), rs_smem(R, NZ, 1, bs));
}
"""


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    """The kernel's own sizes: constants, elements of x, bytes of a block with a table of one row."""
    import os
    import subprocess

    from conftest import ROOT
    from h2_b200 import build
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("layout")
    (d / "layout.cu").write_text(LAYOUT)
    subprocess.run([nvcc, "-std=c++17", "-O0", *build.ARCH, "-I", os.path.join(ROOT, "h2_b200", "csrc"),
                    str(d / "layout.cu"), "-o", str(d / "layout")], check=True, capture_output=True)
    out = subprocess.run([str(d / "layout")], check=True, capture_output=True, text=True).stdout.splitlines()
    consts = dict(zip(("pitch", "box", "row", "most", "warps"), map(int, out[0].split())))
    sizes = {tuple(v[:3]): tuple(v[3:]) for v in (list(map(int, line.split())) for line in out[1:])}
    return consts, sizes


@pytest.mark.parametrize("NZ", [1, 2, 9, 29, 30, 31, 32, 59, 60])
def test_shared_memory_layout(layout, NZ):
    """x, the table of the tile's classes, b and the classes lie one behind the other inside the block's shared memory,
    for every split; the neighbours of every cell lie inside x, the planes of zeros around it included."""
    consts, sizes = layout
    assert consts["pitch"] == 34 and consts["box"] == BOX
    np_ = 1 if NZ <= 30 else 2
    for R in range(1, (8 if np_ == 1 else 4) + 1):
        bs = b_shared(R, np_)
        x, one = sizes[R, NZ, int(bs)]
        P, PL = consts["pitch"], 2 * R * consts["pitch"]
        planes = (NZ + 1) // 2 * 2
        first = PL  # X[0], plane 0
        # the lowest element that a cell reads: the plane below the first, colour 0, beside position 0
        assert first - PL + 0 * P + 0 >= 0
        # the highest: the plane above the last, colour 1, last row, beside position 31
        assert first + planes * PL + R * P + (R - 1) * P + 1 + 32 == x - 1
        # messages written beside a row: 0 or 33 positions on from the cell beside its first position
        assert first + (planes - 1) * PL + R * P + (R - 1) * P + 33 < first + planes * PL
        warps = -(-NZ // (2 * np_))
        assert warps <= consts["warps"] and warps * np_ * 2 <= planes + 2
        tail = planes // 2 * 2 * R * 32 * (4 + (16 if bs else 0))
        assert one == 8 * (x + consts["row"]) + tail
        # a table row for 600 classes at least, beside the row of the cells without a class
        rows = (232448 - 512 - (one - 8 * consts["row"])) // (8 * consts["row"])
        assert rows >= 601, (R, rows)
    if NZ == 30:
        # with b in shared memory tiles of 6 rows would have room for 152 classes
        x, one = sizes[6, 30, 1]
        assert (232448 - 512 - (one - 80)) // 80 - 1 == 152

"""Index arithmetic of the pipelined compress kernels, checked on the CPU.
Mirrors csrc/wide_stream.cuh: the dealing of a step's quads to the threads
(conversions and 128-byte runs), the operand and tile stores, the shuffled
4 x 4 transpose, and the shared memory of the resident CTAs."""
import pytest

CHUNK = 64
SBO = CHUNK // 4 * 128


def core_offset(row, k):
    return (row // 8) * SBO + (k // 4) * 128 + (row % 8) * 16 + (k % 4) * 4


def threads(kp):
    return 256 if kp == 64 else 512


def direct(kp, t, b):
    block = t // 32 + b * (threads(kp) // 32)
    return block // 4 * 8 + t % 8, block % 4 * 4 + t % 32 // 8


def across(kp, t, b):
    block = t // 32 + b * (threads(kp) // 32)
    return block // (kp // 32) * 4 + t % 4, block % (kp // 32) * 8 + t % 32 // 4


def chunk_run(kp, t, b):
    block = t // 32 + b * (threads(kp) // 32)
    return block // 2 * 4 + t % 32 // 8, block % 2 * 8 + t % 8


def row_run(kp, t, b):
    block, blocks = t // 32 + b * (threads(kp) // 32), kp // 32
    return block // blocks * 4 + t % 32 // 8, block % blocks * 8 + t % 8


def direct_at(r, q):
    return r * (CHUNK // 4) + (q ^ (r & 7))


def across_at(kp, r, q):
    return r * (kp // 4) + (q ^ (2 * (r & 3)))


def conflict(offsets):
    """Wavefronts of a 16-byte access over those of a conflict-free one."""
    worst = 0
    for phase in range(0, 32, 8):
        banks = {}
        for offset in offsets[phase:phase + 8]:
            banks.setdefault(offset // 16 % 8, set()).add(offset)
        worst = max(worst, max(len(v) for v in banks.values()))
    return worst


@pytest.mark.parametrize("kp", [64, 128])
def test_every_quad_is_dealt_once(kp):
    n, steps = threads(kp), 4
    for deal in (direct, chunk_run):
        cells = [deal(kp, t, b) for t in range(n) for b in range(steps)]
        assert sorted(cells) == [(r, q) for r in range(kp) for q in range(16)]
    for deal in (across, row_run):
        cells = [deal(kp, t, b) for t in range(n) for b in range(steps)]
        assert sorted(cells) == [(r, q) for r in range(64) for q in range(kp // 4)]
    assert sorted(direct_at(r, q) for r in range(kp) for q in range(16)) == list(range(16 * kp))
    assert (sorted(across_at(kp, r, q) for r in range(64) for q in range(kp // 4))
            == list(range(16 * kp)))
    per_thread = (kp // 4) * (kp // 32) // (n // 32)
    cells = [row_run(kp, t, b) for t in range(n) for b in range(per_thread)]
    assert sorted(cells) == [(r, q) for r in range(kp) for q in range(kp // 4)]


@pytest.mark.parametrize("kp", [64, 128])
@pytest.mark.parametrize("states", [36, 60, 64, 68, 100, 124, 128])
def test_operands_are_whole_and_in_bounds(kp, states):
    if not kp - 64 < states <= kp:
        return
    part = kp * CHUNK * 4
    for d0 in range(0, kp, CHUNK):
        rows = set()
        for t in range(threads(kp)):
            for b in range(4):
                r, q = direct(kp, t, b)
                if r < states:
                    assert core_offset(r, 4 * q) + 16 <= part
                    rows.add((r, 4 * q))
        assert rows == {(r, d) for r in range(states) for d in range(0, 64, 4)}
        columns = set()
        for t in range(threads(kp)):
            for b in range(4):
                d, q = across(kp, t, b)
                if 4 * q < states:  # after the transpose
                    r, d = 4 * q + t % 4, d - d % 4
                    assert r < states and core_offset(r, d) + 16 <= part
                    columns.add((r, d))
        assert columns == {(r, d) for r in range(states) for d in range(0, 64, 4)}


@pytest.mark.parametrize("kp", [64, 128])
def test_bank_conflicts(kp):
    for w in range(threads(kp) // 32):
        lanes = range(32 * w, 32 * w + 32)
        for b in range(4):
            cells = [direct(kp, t, b) for t in lanes]
            assert conflict([core_offset(r, 4 * q) for r, q in cells]) == 1
            cells = [across(kp, t, b) for t in lanes]
            assert conflict([core_offset(r, 4 * q) for r, q in cells]) == 2
            stored = [(4 * q + t % 4, r - r % 4) for t, (r, q) in zip(lanes, cells)]
            assert conflict([core_offset(r, d) for r, d in stored]) <= 2
            assert conflict([16 * direct_at(*c) for c in
                             (direct(kp, t, b) for t in lanes)]) == 1
            assert conflict([16 * across_at(kp, *c) for c in cells]) == 1
            for deal in (chunk_run, row_run):
                cells = [deal(kp, t, b) for t in lanes]
                assert conflict([16 * direct_at(r, q % 16) for r, q in cells]) == 1
                assert conflict([16 * across_at(kp, r, q) for r, q in cells]) == 1
                assert conflict([(r * (kp // 4) + (q ^ (r & 7))) * 16 for r, q in cells]) == 1
                for first in range(0, 32, 8):  # a quarter warp: one run of 128 bytes
                    run = cells[first:first + 8]
                    assert len({r for r, _ in run}) == 1
                    assert [q - run[0][1] for _, q in run] == list(range(8))
    # A row per thread, the same quad of 32 consecutive rows.
    for q in range(kp // 4):
        assert conflict([(r * (kp // 4) + (q ^ (r & 7))) * 16 for r in range(32)]) == 1


def test_shuffled_transpose():
    v = [[10 * lane + j for j in range(4)] for lane in range(4)]
    step = [row[:] for row in v]
    for lane in range(4):
        partner, odd = lane ^ 1, lane & 1
        sent = (v[partner][0], v[partner][2]) if partner & 1 else (v[partner][1], v[partner][3])
        if odd:
            step[lane][0], step[lane][2] = sent
        else:
            step[lane][1], step[lane][3] = sent
    out = [row[:] for row in step]
    for lane in range(4):
        partner, high = lane ^ 2, lane & 2
        sent = step[partner][:2] if partner & 2 else step[partner][2:]
        if high:
            out[lane][:2] = sent
        else:
            out[lane][2:] = sent
    assert out == [[v[j][lane] for j in range(4)] for lane in range(4)]


@pytest.mark.parametrize("kp,reverse", [(64, False), (64, True), (128, False), (128, True)])
def test_resident_ctas_fit(kp, reverse):
    part, slot = kp * CHUNK * 4, 4 * threads(kp) * 16
    size = 4 * part + (3 if reverse else 2) * slot + 2 * kp * 4
    resident = 2 if kp == 64 else 1
    assert size + 512 <= 227 * 1024 and resident * (size + 512 + 1024) <= 228 * 1024
    assert 2 * kp * kp * 4 <= 4 * part  # the two epilogue tiles
    columns = 128 if kp == 64 else 512
    assert resident * columns <= 512 and (kp // CHUNK + 1) * kp <= columns and 2 * kp <= columns

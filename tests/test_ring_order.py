"""The ring order of mega_ring.cu, restated in Python: the producer warps enumerate a CTA's items of a streaming MATVEC phase in one
order (mr_item), the consumer warps take groups of two rows round-robin and walk the same items by index arithmetic (phase_matvec_ring).  Both
sides must agree on which (group, segment) sits in item e, and every (unit, virtual row, segment) must be produced exactly once.  This test pins the
arithmetic (a change on one side of the CUDA file has to be mirrored here and on the other side); the CUDA code itself is checked on the GPU by the
bit-identity tests (tests/test_gpu_runner.py, tests/test_gpu_ring_rows.py)."""
import pytest

MK_SEG = 4
WARPS = 16
GRID = 148


def geo(m, n_mats, k, epilogue, cta, grid=GRID):
    """mr_geo: rows of the phase that belong to CTA `cta`, one contiguous run; a group is two neighbouring rows of one matrix (gate and up: in turn)."""
    nb = k // 32
    gr = (nb + 31) // 32
    nseg = (gr + MK_SEG - 1) // MK_SEG
    pair = epilogue == 2
    m_cat = m if pair else m * n_mats
    if epilogue == 3:
        rpc = ((m_cat + grid - 1) // grid + 3) & ~3
        first = cta * rpc
        n_rows = min(rpc, max(0, m_cat - first))
        most = rpc
    else:
        each, more = divmod(m_cat, grid)
        first = cta * each + min(cta, more)
        n_rows = each + (1 if cta < more else 0)
        most = (each + (1 if more else 0)) * (2 if pair else 1)
    return dict(most=most, nb=nb, nseg=nseg, V=2 if pair else 1, n_units=n_rows, first=first, stride=1, groups=(n_rows + 1) // 2 * (2 if pair else 1))


def rows_of(g, P):
    """the (unit, virtual row) pairs of group P"""
    u, v = (P & ~1, P & 1) if g["V"] == 2 else (2 * P, 0)
    return [(x, v) for x in (u, u + 1) if x < g["n_units"]]


def producer_order(g):
    """mr_item: item index j -> [(unit, virtual row, segment)] of its one or two rows."""
    out = []
    for j in range(g["groups"] * g["nseg"]):
        P, sg = divmod(j, g["nseg"])
        out.append([(u, v, sg) for u, v in rows_of(g, P)])
    return out


def consumer_walk(g):
    """phase_matvec_ring: for every pair of warps the list of (item index, [(unit, virtual row, segment)]) it consumes, in order."""
    walks, nseg, duos = [], g["nseg"], WARPS // 2
    part_bytes = g["most"] * 132 if nseg == 1 else g["most"] * nseg * 128            # cc_mega_ring_layout
    split = 1 < nseg <= duos and part_bytes <= (57344 if nseg > 4 else 30720)        # warps keep to one segment
    for duo in range(duos):
        s0, ns = (duo % nseg, 1) if split else (0, nseg)
        p0, dp = (duo // nseg, (duos - s0 + nseg - 1) // nseg) if split else (duo, duos)
        walk, e = [], p0 * nseg + s0
        for P in range(p0, g["groups"], dp):
            for s in range(ns):
                walk.append((e, [(u, v, s0 + s) for u, v in rows_of(g, P)]))
                e += 1 if s + 1 < ns else (dp - 1) * nseg + (nseg if split else 1)
        walks.append(walk)
    return walks


SHAPES = [  # (rows per matrix, matrices, k, epilogue)
    (4096, 3, 4096, 0), (4096, 1, 4096, 1), (11008, 2, 4096, 2), (4096, 1, 11008, 1), (32000, 1, 4096, 0),      # Llama-2-7B, one GPU
    (4096, 1, 2048, 3), (4096, 1, 5504, 3), (16000, 1, 4096, 3),                                                    # shards at N = 2 (exchange phases)
    (512, 3, 4096, 0), (4096, 1, 512, 3), (1376, 2, 4096, 2), (4096, 1, 1376, 3), (4000, 1, 4096, 3),               # shards at N = 8
    (4096, 1, 14336, 1), (8192, 1, 28672, 1), (256000, 1, 8192, 0), (28672, 2, 8192, 2),                          # four segments, seven, and more rows than their sums find room for
    (8192, 1, 18432, 1), (8192, 1, 24576, 1), (8192, 1, 29568, 1), (12288, 1, 32768, 1), (148, 1, 65536, 1),      # five, six, eight with room and without, sixteen
    (34386, 1, 4096, 0), (4440, 2, 14336, 2),                                                                      # CTAs on both sides of the room for lanes' sums
    (288, 3, 288, 0), (288, 1, 288, 1), (768, 2, 288, 2), (288, 1, 768, 1), (32000, 1, 288, 0),                     # tinyllamas-15M (ragged groups)
]


@pytest.mark.parametrize("m,n_mats,k,epilogue", SHAPES)
def test_producer_and_consumers_agree_on_the_ring_order(m, n_mats, k, epilogue):
    covered_rows = set()
    for cta in (0, 1, 37, 146, 147):
        g = geo(m, n_mats, k, epilogue, cta)
        order = producer_order(g)
        # every (unit, virtual row, segment) of the CTA exactly once
        want = {(u, v, s) for u in range(g["n_units"]) for v in range(g["V"]) for s in range(g["nseg"])}
        got = [x for item in order for x in item]
        assert len(got) == len(want) and set(got) == want
        seen = []
        for walk in consumer_walk(g):
            for e, rows in walk:
                assert order[e] == rows, (cta, e, order[e], rows)
                seen.append(e)
        assert sorted(seen) == list(range(len(order)))                # the consumers release every slot exactly once
        covered_rows.update(g["first"] + u * g["stride"] for u in range(g["n_units"]))
    assert covered_rows                                               # (the sampled CTAs own rows)


@pytest.mark.parametrize("m,n_mats,k,epilogue", SHAPES)
def test_no_cta_has_more_rows_than_the_layout_in_shared_memory_allows(m, n_mats, k, epilogue):
    """the host lays shared memory out (and decides whether lanes' sums have room) by the CTA with the most rows (cc_mega_ring_layout)"""
    geos = [geo(m, n_mats, k, epilogue, cta) for cta in range(GRID)]
    rows = -(-(m if epilogue == 2 else m * n_mats) // GRID)
    host = 2 * rows if epilogue == 2 else (rows + 3) & ~3 if epilogue == 3 else rows
    assert {g["most"] for g in geos} == {host}
    assert max(g["n_units"] * g["V"] for g in geos) <= host


@pytest.mark.parametrize("m,n_mats,k,epilogue", SHAPES)
def test_every_row_of_a_phase_belongs_to_exactly_one_cta(m, n_mats, k, epilogue):
    rows = []
    for cta in range(GRID):
        g = geo(m, n_mats, k, epilogue, cta)
        rows += [g["first"] + u * g["stride"] for u in range(g["n_units"])]
    m_cat = m if epilogue == 2 else m * n_mats
    assert sorted(rows) == list(range(m_cat))


def test_items_that_come_free_together_are_issued_by_different_warps():
    """mr_producer: thread 3 * lane + warp owns item t mod 96; of any ring's worth of neighbouring items no warp has more than a third (its lanes issue one after another)"""
    owner = {lane * 3 + warp: warp for warp in range(3) for lane in range(32)}
    assert sorted(owner) == list(range(96))
    for first in range(96):
        for items in (8, 17, 24, 48):
            share = [sum(owner[e % 96] == w for e in range(first, first + items)) for w in range(3)]
            assert max(share) <= -(-items // 3), (first, items, share)

"""The steps of the device's entropy coding that whole encodes of test size do not bring to their limits,
called one by one: a frame whose token total passes 32 bits, a frame that goes through in several groups of
tiles, and CDF lists whose segments were adapted from a state that was not the true one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U32, I32, P = C.c_uint32, C.c_int32, C.c_void_p
GROUP_TOKENS = 256 * 64  # what a tile's tokens are padded to


class Geom(C.Structure):
    _fields_ = [(n, I32) for n in ("nbx", "nby", "sub", "sb_cols", "sb_rows", "tile_w8", "tile_h8", "tcols",
                                   "trows")] + [("max_tokens", U32)]


class Input(C.Structure):
    _fields_ = [("mode", P), ("tx", P), ("lv", P * 3)]


class Totals(C.Structure):
    _fields_ = [(n, U32) for n in ("tokens", "digits", "bytes", "groups")]


class Group(C.Structure):
    _fields_ = [("tile0", I32), ("ntiles", I32), ("tokens", U32)]


TILE = np.dtype([(n, np.uint32) for n in ("base", "ntok", "shift", "digit", "byte", "nbytes")])


class Steps:
    """csrc/stream.h over one frame, on the default stream."""

    def __init__(self, lib, torch, nbx, nby, sub, tile8, max_tokens):
        self.torch, self.n = torch, I32(0)
        up = lambda a, b: (a + b - 1) // b  # noqa: E731
        self.g = Geom(nbx, nby, sub, up(nbx, 8), up(nby, 8), tile8[0], tile8[1],
                      up(nbx, tile8[0]), up(nby, tile8[1]), max_tokens)
        self.nt = self.g.tcols * self.g.trows

        def bind(name, res, *args):
            f = getattr(lib, name)
            f.restype, f.argtypes = res, args
            return f

        geom, inp, tot, grp, n = C.POINTER(Geom), C.POINTER(Input), C.POINTER(Totals), C.POINTER(Group), C.POINTER(I32)
        self._plan_bytes = bind("_ZN3mth17stream_plan_bytesERKNS_10StreamGeomE", C.c_size_t, geom)
        self._token_bytes = bind("_ZN3mth18stream_token_bytesERKNS_10StreamGeomEj", C.c_size_t, geom, U32)
        self._digit_bytes = bind("_ZN3mth18stream_digit_bytesERKNS_12StreamTotalsE", C.c_size_t, tot)
        self._count = bind("_ZN3mth12stream_countERKNS_10StreamGeomERKNS_11StreamInputEPvP11CUstream_stPi", C.c_int,
                           geom, inp, P, P, n)
        self._place = bind("_ZN3mth12stream_placeERKNS_10StreamGeomEPvP11CUstream_stPi", C.c_int, geom, P, P, n)
        self._counts = bind("_ZN3mth13stream_countsERKNS_10StreamGeomEPv", P, geom, P)
        self._totals = bind("_ZN3mth13stream_totalsERKNS_10StreamGeomEPv", P, geom, P)
        self._tiles = bind("_ZN3mth12stream_tilesERKNS_10StreamGeomEPv", P, geom, P)
        self._group = bind("_ZN3mth12stream_groupEPKNS_10StreamTileEii", Group, P, I32, I32)
        self._trace = bind("_ZN3mth12stream_traceERKNS_10StreamGeomERKNS_11StreamInputEPvS6_RKNS_11StreamGroupEPKvb"
                           "P11CUstream_stPi", C.c_int, geom, inp, P, P, grp, P, C.c_bool, P, n)
        self._ranges = bind("_ZN3mth13stream_rangesERKNS_10StreamGeomEPvS3_RKNS_11StreamGroupEPKiPKhP11CUstream_stPi",
                            C.c_int, geom, P, P, grp, P, P, P, n)
        self._bytes = bind("_ZN3mth12stream_bytesERKNS_10StreamGeomEPvS3_RKNS_11StreamGroupES3_RKNS_12StreamTotalsEj"
                           "P11CUstream_stPi", P, geom, P, P, grp, P, tot, U32, P, n)
        table = bind("_ZN3mth16stream_cdf_tableEii", P, I32, I32)
        self.cdfs = np.ctypeslib.as_array((C.c_uint16 * 4096).from_address(table(1, sub))).reshape(256, 16).copy()
        self.d_cdfs = torch.from_numpy(self.cdfs.view(np.int16)).cuda()
        self.plan = self.buffer(self._plan_bytes(self.g))

    def buffer(self, n):
        return self.torch.zeros(max(int(n), 1), dtype=self.torch.uint8, device="cuda")

    def at(self, buf, address, count, dtype):
        """`count` entries of a device buffer from `address` on."""
        o = address - buf.data_ptr()
        return buf[o:o + count * np.dtype(dtype).itemsize]

    def read(self, buf, address, count, dtype):
        return self.at(buf, address, count, dtype).cpu().numpy().view(dtype)

    def totals(self):
        return Totals.from_buffer_copy(self.read(self.plan, self._totals(self.g, self.plan.data_ptr()), 16, np.uint8))

    def tiles(self):
        return self.read(self.plan, self._tiles(self.g, self.plan.data_ptr()), self.nt, TILE)

    def place(self, counts):
        slots = self.at(self.plan, self._counts(self.g, self.plan.data_ptr()), len(counts), np.uint32)
        slots.copy_(self.torch.from_numpy(counts.view(np.uint8)))
        assert self._place(self.g, self.plan.data_ptr(), None, self.n) == 0
        return self.totals(), self.tiles()

    def load(self, mode, tx, levels):
        up = lambda a: self.torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.dev = [up(mode), up(tx)] + [up(v) for v in levels]
        self.inp = Input(self.dev[0].data_ptr(), self.dev[1].data_ptr(), (P * 3)(*[d.data_ptr() for d in self.dev[2:]]))
        assert self._count(self.g, self.inp, self.plan.data_ptr(), None, self.n) == 0
        tot, tiles = self.totals(), self.tiles()
        self.tokens = self.buffer(self._token_bytes(self.g, tot.tokens))
        groups, t = [], 0
        while t < self.nt:
            groups.append(self._group(tiles.ctypes.data, self.nt, t))
            t += groups[-1].ntiles
        assert len(groups) == tot.groups and max(g.tokens for g in groups) == tot.tokens
        return groups

    def trace(self, grp, updating=True):
        assert self._trace(self.g, self.inp, self.plan.data_ptr(), self.tokens.data_ptr(), grp, self.d_cdfs.data_ptr(),
                           updating, None, self.n) == 0

    def payloads(self, grp, bits, grid):
        d_bits, d_grid = (self.torch.from_numpy(np.array(a)).cuda() for a in ([bits], grid))
        d_bits = d_bits.int()
        args = (self.g, self.plan.data_ptr(), self.tokens.data_ptr(), grp)
        assert self._ranges(*args, d_bits.data_ptr(), d_grid.data_ptr(), None, self.n) == 0
        tot, tiles = self.totals(), self.tiles()[grp.tile0:grp.tile0 + grp.ntiles]
        digits = self.buffer(self._digit_bytes(tot))
        out = self._bytes(*args, digits.data_ptr(), tot, int(tiles["nbytes"].max()), None, self.n)
        assert out
        data = self.read(digits, out, tot.bytes, np.uint8)
        return [data[t["byte"]:t["byte"] + t["nbytes"]].tobytes() for t in tiles]


@pytest.mark.parametrize("top,max_tokens", [(9_000_000, 1 << 30), (9_000_000, 1), (30_000, 1 << 30), (30_000, 1 << 22)])
def test_a_token_total_past_32_bits_is_laid_out_in_groups_of_tiles(mt_lib, cuda, top, max_tokens):
    s = Steps(mt_lib.load(), cuda, 45, 19, 0, (16, 8), max_tokens)
    counts = np.random.default_rng(top).integers(top // 3, top, 3 * 45 * 19, dtype=np.uint32)
    tot, tiles = s.place(counts)
    assert top < 1_000_000 or int(counts.sum(dtype=np.uint64)) > 1 << 32
    at = base = most = 0
    groups = 1
    for t in range(s.nt):
        w, h = min(16, 45 - t % s.g.tcols * 16), min(8, 19 - t // s.g.tcols * 8)
        n = int(counts[at:at + 3 * w * h].sum(dtype=np.uint64))
        at += 3 * w * h
        padded = -(-n // GROUP_TOKENS) * GROUP_TOKENS
        if base and base + padded > max_tokens:
            base, groups = 0, groups + 1
        assert (int(tiles["base"][t]), int(tiles["ntok"][t])) == (base, n), t
        base += padded
        most = max(most, base)
    assert (tot.tokens, tot.groups) == (most, groups)


@pytest.mark.parametrize("sub", [0, 2])
@pytest.mark.parametrize("max_tokens,ngroups", [(1, 15), (150_000, None)])
def test_groups_of_tiles_give_the_bytes_of_one(mt_lib, cuda, sub, max_tokens, ngroups):
    rng = np.random.default_rng(sub + 5)
    nbx, nby = 37, 21
    nb, cl = nbx * nby, 16 if sub else 64

    def levels(n):
        v = rng.integers(-40, 41, (nb, n)) * (rng.random((nb, n)) < rng.random((nb, 1)))
        return v.astype(np.int32)

    frame = (rng.integers(0, 13, nb).astype(np.uint8), rng.integers(0, 7, nb).astype(np.uint8),
             [levels(64), levels(cl), levels(cl)])
    grid = rng.integers(0, 4, 15).astype(np.uint8)
    got = []
    for limit in (1 << 30, max_tokens):
        s = Steps(mt_lib.load(), cuda, nbx, nby, sub, (8, 8), limit)
        groups, out = s.load(*frame), []
        for grp in groups:
            s.trace(grp)
            out += s.payloads(grp, 2, grid)
        got.append(out)
        if limit == 1 << 30:
            assert len(groups) == 1
    assert len(groups) > 1 and ngroups in (None, len(groups))
    assert len(got[0]) == 15 and got[0] == got[1]


SEG, WARM, TXTP = 1024, 2, 66  # entries of a segment, warm-up segments, the tx-type CDF of DC_PRED


class Cdf:
    """update_cdf on an inverse CDF of n symbols, one symbol at a time."""

    def __init__(self, entries, n, done=0):
        self.c, self.n, self.done = [int(v) for v in entries[:n - 1]], n, done

    def copy(self):
        return Cdf(self.c, self.n, self.done)

    def code(self, s):
        """The store of symbol s (fl >> 6, fh >> 6 << 10, n - s << 20), then the update."""
        c = self.c
        word = ((c[s - 1] if s else 32768) >> 6) | ((c[s] if s < self.n - 1 else 0) >> 6) << 10 | (self.n - s) << 20
        rate = 3 + min(self.n >> 1, 2) + (self.done >> 4)
        for e in range(self.n - 1):
            c[e] += ((32768 - c[e]) >> rate) if s > e else -(c[e] >> rate)
        self.done = min(self.done + 1, 32)
        return word


def test_segments_that_started_wrong_are_redone(mt_lib, cuda):
    """A list of 260 segments (two turns of 256) of a repeated pattern, on which
    two states need not meet: most segments are adapted from a wrong state at
    first, many in a row, and every store still is the one of the serial
    adaptation."""
    nbx, nby = 512, 520
    nb = nbx * nby
    y, x = np.mgrid[0:nby, 0:nbx]
    z = sum(((x >> i) & 1) << (2 * i) | ((y >> i) & 1) << (2 * i + 1) for i in range(3))
    pos = ((y >> 3) * (nbx // 8) + (x >> 3)) * 64 + z
    seq = np.arange(nb) % 3 * 3  # the types' symbols, in coding order
    luma = np.zeros((nb, 64), np.int32)
    luma[:, 0] = 1
    none = np.zeros((nb, 16), np.int32)
    s = Steps(mt_lib.load(), cuda, nbx, nby, 2, (nbx, nby), 1 << 30)
    (grp,) = s.load(np.zeros(nb, np.uint8), seq[pos].astype(np.uint8).ravel(), [luma, none, none])
    s.trace(grp)
    n = grp.tokens  # the buffer starts with the stores, an index and the tokens (4, 4 and 2 bytes each)
    raw = s.tokens[:10 * n].cpu().numpy()
    stores, tok = raw[:4 * n].view(np.uint32), raw[8 * n:].view(np.uint16)[:s.tiles()["ntok"][0]]
    at = np.flatnonzero((tok & 255) == TXTP)
    assert np.array_equal(tok[at] >> 8, seq) and len(seq) > 256 * SEG
    cdf = Cdf(s.cdfs[TXTP], int(s.cdfs[TXTP][15]))
    want, before = np.zeros(nb, np.uint32), []
    symbols = seq.tolist()
    for i, sym in enumerate(symbols):
        if i % SEG == 0:
            before.append(cdf.copy())
        want[i] = cdf.code(sym)
    # the segments of the first 24 whose warmed-up state is not the true one
    wrong = []
    rest = (1 << (5 + min(cdf.n >> 1, 2))) - 1
    for k in range(WARM + 2, 24):
        first = symbols[SEG:(k - WARM) * SEG]
        guess = before[1].copy()
        for e in range(cdf.n - 1):
            if max(first) > e and guess.c[e] < rest:
                guess.c[e] = rest
            if min(first) <= e and guess.c[e] > 32768 - rest:
                guess.c[e] = 32768 - rest
        for sym in symbols[(k - WARM) * SEG:k * SEG]:
            guess.code(sym)
        wrong.append(guess.c != before[k].c)
    assert sum(wrong) > 8 and any(a and b for a, b in zip(wrong, wrong[1:]))
    assert np.array_equal(stores[at], want)

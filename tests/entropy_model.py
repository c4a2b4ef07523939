"""Model of the bookkeeping of the block-parallel JPEG entropy kernels (aeon_b200/csrc/jpeg_entropy.cu): segments, guessed
entry states, checkpoints, rounds of re-decoding with an early exit at a checkpoint passed in a noted state, block counts,
and the storing pass dealt out in pieces between checkpoints.  Plain python over the bit string of a baseline JPEG; the
kernel follows the same steps (it takes AC symbols in pairs where the first cannot reach the place a run looks for, which comes to the
same).  `simulate` returns what the kernel would count and every inconsistency it finds: a segment
whose block count differs from the true one, a piece that would start at a wrong block number or meet an invalid symbol, a
checkpoint the storing pass needs that no run has written.  Test infrastructure only."""
import numpy as np

from oracle import jpeg as J

NCHECK = 3           # checkpoints inside a segment
MIN_SEGMENT = 160    # bytes


def _parse(blob):
    """Huffman tables, sampling factors, table selectors, picture size and the offset of the entropy-coded data."""
    dc = {0: J._Huff(*J.STD_DC_LUMA), 1: J._Huff(*J.STD_DC_CHROMA)}
    ac = {0: J._Huff(*J.STD_AC_LUMA), 1: J._Huff(*J.STD_AC_CHROMA)}
    comps, width, height, p = [], 0, 0, 2
    while True:
        assert blob[p] == 0xFF
        marker = blob[p + 1]
        p += 2
        length = (blob[p] << 8) | blob[p + 1]
        seg = blob[p + 2:p + length]
        if marker == 0xC4:
            q = 0
            while q < len(seg):
                tc, th = seg[q] >> 4, seg[q] & 15
                bits = list(seg[q + 1:q + 17])
                vals = list(seg[q + 17:q + 17 + sum(bits)])
                q += 17 + sum(bits)
                (ac if tc else dc)[th] = J._Huff(bits, vals)
        elif marker == 0xC0:
            height, width = (seg[1] << 8) | seg[2], (seg[3] << 8) | seg[4]
            comps = [(seg[7 + 3 * i] >> 4, seg[7 + 3 * i] & 15) for i in range(seg[5])]
        elif marker == 0xDA:
            selectors = [(seg[2 + 2 * i] >> 4, seg[2 + 2 * i] & 15) for i in range(seg[0])]
            return p + length, dc, ac, comps, selectors, width, height
        p += length


class _Stream:
    """A baseline stream without its stuffed bytes, and what the true decoder makes of it."""

    def __init__(self, blob):
        start, dc, ac, comps, selectors, width, height = _parse(blob)
        scan = blob[start:-2]
        clean, i = bytearray(), 0
        while i < len(scan):                               # the copy without stuffed bytes
            clean.append(scan[i])
            i += 2 if scan[i] == 0xFF and i + 1 < len(scan) and scan[i + 1] == 0 else 1
        self.scan_bytes, self.clean_bytes, self.total_bit = len(scan), len(clean), len(clean) * 8
        bits = np.unpackbits(np.frombuffer(bytes(clean) + b"\0" * 16, np.uint8)).astype(np.int32)
        window = np.zeros(len(bits) - 16, np.int32)        # the 16 bits from every position on
        for k in range(16):
            window = window << 1 | bits[k:len(bits) - 16 + k]
        self._window = window.tolist()

        hmax, vmax = max(c[0] for c in comps), max(c[1] for c in comps)
        block_comp = []                                    # component of every block of an MCU
        for ci, (h, v) in enumerate(comps):
            block_comp += [ci] * (h * v if len(comps) > 1 else 1)
        self.bpm = len(block_comp)
        mcux = -(-width // (8 * hmax)) if len(comps) > 1 else -(-width // 8)
        mcuy = -(-height // (8 * vmax)) if len(comps) > 1 else -(-height // 8)
        self.total_blocks = mcux * mcuy * self.bpm
        self._dc = [self._codes(dc[selectors[c][0]], True) for c in block_comp]    # per block of an MCU
        self._ac = [self._codes(ac[selectors[c][1]], False) for c in block_comp]

        self.starts, self.block_ends = [], []              # bits at which a symbol / the last symbol of a block starts
        p, b, k, done = 0, 0, 0, 0
        while done < self.total_blocks:
            taken, _, advance = self.symbol(p, b, k)
            assert advance != 127
            self.starts.append(p)
            if k + advance >= 64:
                self.block_ends.append(p)
            p, k = p + taken, k + advance
            if k >= 64:
                k, done, b = 0, done + 1, (b + 1) % self.bpm
        self.block_ends = np.array(self.block_ends)

    @staticmethod
    def _codes(table, is_dc):
        """(bits taken, value bits, advance of the zig-zag index) for every 16 bits a symbol can start with."""
        out = [(16, 0, 127)] * 65536                       # invalid code
        for (length, code), sym in table.lookup.items():
            size, run = sym & 15, sym >> 4
            advance = (1 if run == 0 else 127) if is_dc else (run + 1) if size else (16 if run == 15 else 64)
            first = code << (16 - length)
            out[first:first + (1 << (16 - length))] = [(length + size, size, advance)] * (1 << (16 - length))
        return out

    def symbol(self, p, b, k):
        return (self._dc if k == 0 else self._ac)[b][self._window[p]]


def simulate(blob, threads=512, checkpoint_past_end=False):
    """Runs the kernel's passes over one stream.  `checkpoint_past_end` restores the rule that once let a run note (or fall
    into step at) a checkpoint lying within a symbol's reach past the end of the last segment."""
    stream = _Stream(blob)
    bpm, total_bit, total_blocks, block_ends, symbol = stream.bpm, stream.total_bit, stream.total_blocks, stream.block_ends, stream.symbol

    seg = max((-(-stream.clean_bytes // threads) + 3) & ~3, MIN_SEGMENT)
    deals = max(((NCHECK + 1) * -(-stream.clean_bytes // seg) * 4 + 3 * threads) // (4 * threads), 1)   # rounds of the storing pass
    seg = max(seg, ((NCHECK + 1) * stream.clean_bytes // (deals * threads) + 4) & ~3)                   # no nearly empty last one
    nseg = -(-stream.clean_bytes // seg)
    step = seg * 8 // (NCHECK + 1)

    def run(p, b, k, pend, notes, compare, old_blocks, storing=False):
        blocks, bad, merged, j = 0, False, False, 0
        check_at = None
        if not storing and (checkpoint_past_end or notes["first"] < pend):
            check_at = notes["first"]
        while p < pend:
            taken, size, advance = symbol(p, b, k)
            if storing and (advance == 127 or (k != 0 and size and k + advance - 1 > 63)):
                bad = True
            p, k = p + taken, k + advance
            if k >= 64:
                k, blocks, b = 0, blocks + 1, (b + 1) % bpm
            if check_at is not None and p >= check_at:
                assert p - check_at <= 30
                key = (p - check_at) << 10 | b << 6 | k
                if compare and notes["key"][j] == key:     # in step with the remembered run
                    was = notes["blocks"][j]
                    for later in range(j, NCHECK):
                        if notes["blocks"][later] is not None:
                            notes["blocks"][later] += blocks - was
                    blocks += old_blocks - was
                    merged = True
                    break
                notes["key"][j], notes["blocks"][j] = key, blocks
                j += 1
                more = j < NCHECK and (checkpoint_past_end or check_at + step < pend)
                check_at = check_at + step if more else None
        return p, b, k, blocks, bad, merged

    segments = []
    for t in range(nseg):                                  # first pass: guessed entry states
        first, last = t * seg * 8, min(total_bit, (t + 1) * seg * 8)
        notes = {"first": first + step, "key": [None] * NCHECK, "blocks": [None] * NCHECK}
        p, b, k, blocks, _, _ = run(first, 0, 0, last, notes, False, 0)
        segments.append({"first": first, "last": last, "notes": notes, "entry": (first, 0, 0), "exit": (p, b, k), "count": blocks})
    rounds = 0
    while True:                                            # rounds: the left neighbour's exit state is the entry state
        rounds += 1
        candidates = [None] + [segments[t - 1]["exit"] for t in range(1, nseg)]
        again = False
        for t in range(1, nseg):
            s = segments[t]
            if candidates[t] != s["entry"]:
                again = True
                p, b, k, blocks, _, merged = run(*candidates[t], s["last"], s["notes"], True, s["count"])
                s["entry"], s["count"] = candidates[t], blocks
                if not merged:
                    s["exit"] = (p, b, k)
        if not again:
            break
        assert rounds <= nseg

    problems = []
    counted = sum(s["count"] for s in segments)
    if counted != total_blocks:
        problems.append(("counted", counted, total_blocks))
    first_block = 0
    for t, s in enumerate(segments):                       # the storing pass, piece by piece
        true_count = int(((block_ends >= s["entry"][0]) & (block_ends < s["last"])).sum())
        if true_count != s["count"]:
            problems.append(("segment count", t, s["count"], true_count))
        for piece in range(NCHECK + 1):
            at = s["first"] + piece * step
            if at >= s["last"]:
                continue
            if piece == 0:
                (p0, b0, k0), before = s["entry"], 0
            else:
                key = s["notes"]["key"][piece - 1]
                if key is None:
                    problems.append(("unwritten checkpoint", t, piece))
                    continue
                p0, b0, k0, before = at + (key >> 10), key >> 6 & 15, key & 63, s["notes"]["blocks"][piece - 1]
            if p0 < total_bit and int((block_ends < p0).sum()) != first_block + before:
                problems.append(("piece block number", t, piece))
            if run(p0, b0, k0, min(s["last"], at + step), None, False, 0, storing=True)[4]:
                problems.append(("piece meets an invalid symbol", t, piece))
        first_block += s["count"]
    return {"bytes": stream.clean_bytes, "segment": seg, "segments": nseg, "rounds": rounds, "counted": counted,
            "total_blocks": total_blocks, "problems": problems}


SPREAD_SEGMENT, SPREAD_CHECKS, SPREAD_GROUP, SPREAD_EXTRA, SPREAD_CAP, SPREAD_PLACES = 128, 4, 16, 256, 1200, 6


def spread_plan(streams, longest, places):
    """Blocks of the cluster of each stream, and the runs a block has room for."""
    segments, blocks = longest // SPREAD_SEGMENT + 1, 8 if streams <= 15 else 4 if streams <= 33 else 2
    assert streams <= 66 and places <= SPREAD_PLACES
    while blocks > 1 and segments * places <= blocks // 2 * 128:
        blocks //= 2
    return blocks, min(SPREAD_CAP, (-(-segments // blocks) + 3) * places)


def simulate_spread(blob, streams=1, extra_room=SPREAD_EXTRA):
    """The same for the kernel that spreads a stream over a cluster of blocks: a run from every place in the MCU for every segment, the
    run that each falls into step with behind its segment, the path from run to run and its short cuts (through a group of segments,
    through a block), and the storing pass in the pieces between known states.  `extra_room`: states a block can note between
    a run's exit and where it falls into step.  Every symbol of the stream has to be stored once, with its block's number."""
    stream = _Stream(blob)
    H, total, symbol = stream.bpm, stream.total_bit, stream.symbol
    C, cap = spread_plan(streams, stream.scan_bytes, H)
    most = C * (cap // H - 2)
    seg = max(SPREAD_SEGMENT, (-(-stream.clean_bytes // most) + SPREAD_CHECKS - 1) // SPREAD_CHECKS * SPREAD_CHECKS)
    bits, step = seg * 8, seg * 8 // SPREAD_CHECKS
    nseg = -(-stream.clean_bytes // seg)
    per = max(-(-nseg // C), 1)
    assert per * H <= cap

    def run(state, until):                                 # state: position, block, index, blocks completed
        p, b, k, blocks = state
        while p < until:
            taken, _, advance = symbol(p, b, k)
            p, k = p + taken, k + advance
            if k >= 64:
                k, b, blocks = 0, (b + 1) % H, blocks + 1
        return p, b, k, blocks

    key, count, state = {}, {}, {}                         # by segment, place, checkpoint
    for s in range(nseg):
        for h in range(H):
            at = (s * bits, h, 0, 0)
            for j in range(SPREAD_CHECKS):
                stop = s * bits + (j + 1) * step
                at = run(at, min(stop, total))
                key[s, h, j] = (at[0] - stop, at[1], at[2]) if stop < total else None
                count[s, h, j], state[s, h, j] = at[3], at

    after, end, extras, noted = {}, {}, [], [0] * C        # after: (run and checkpoint it falls into step with, blocks)
    for s in range(nseg):
        for h in range(H):
            had, k = count[s, h, SPREAD_CHECKS - 1], key[s, h, SPREAD_CHECKS - 1]
            after[s, h] = (None, had)
            if k is None:
                continue
            q, j, stop, last = s + 1, 0, (s + 1) * bits, ("end", s, h)
            at = (stop + k[0], k[1], k[2], 0)
            while True:
                stop += step
                if stop >= total:
                    at = run(at, total)
                    end[last], after[s, h] = total, (None, had + at[3])
                    break
                at = run(at, stop)
                here = (at[0] - stop, at[1], at[2])
                same = [g for g in range(H) if key[q, g, j] == here]
                if same:
                    end[last], after[s, h] = at[0], ((q, same[-1], j), had + at[3] - count[q, same[-1], j])
                    break
                noted[s // per] += 1
                if noted[s // per] <= extra_room:
                    end[last] = at[0]
                    last = ("extra", len(extras))
                    extras.append((s, h, at[0], at[1], at[2], had + at[3]))
                j = (j + 1) % SPREAD_CHECKS
                q += j == 0

    problems = []

    def follow(at, inside):                                # from run to run as long as `inside` holds for its segment
        path = []
        while at[0] is not None and inside(at[0][0]):
            path.append(at)
            to, blocks = after[at[0][:2]]
            at = (to, at[1] + blocks)
        return at, path

    group, through = {}, {}                                # groups count from their block's first segment
    first_of = lambda s: s // per * per + (s % per) // SPREAD_GROUP * SPREAD_GROUP  # noqa: E731
    for s in range(nseg):
        if first_of(s) == s:
            stop = min(s + SPREAD_GROUP, (s // per + 1) * per)
            for h in range(H):
                group[s, h] = follow(((s, h, 0), 0), lambda q: q < stop)[0]

    def hop(at):
        to, blocks = (group if first_of(at[0][0]) == at[0][0] else after)[at[0][:2]]
        return to, at[1] + blocks

    for r in range(C):
        if r * per < nseg:
            for h in range(H):
                at = ((r * per, h, 0), 0)
                while at[0] is not None and at[0][0] < (r + 1) * per:
                    at = hop(at)
                through[r, h] = at
    whole = follow(((0, 0, 0), 0), lambda q: True)
    truth = {at[0][0]: at for at in whole[1]}
    if whole[0][1] < stream.total_blocks:
        problems.append(("counted", whole[0][1], stream.total_blocks))
    for r in range(C):                                     # every block finds its own part of the path by the short cuts
        at, inside = ((0, 0, 0), 0), {}
        while at[0] is not None and at[0][0] < r * per:
            owner = at[0][0] // per
            if at[0][0] == owner * per:
                to, blocks = through[owner, at[0][1]]
                at = (to, at[1] + blocks)
            else:
                at = hop(at)
        while at[0] is not None and at[0][0] < (r + 1) * per:
            inside.setdefault(first_of(at[0][0]), at)
            at = hop(at)
        mine = {}
        for first, at in inside.items():
            stop = min(first + SPREAD_GROUP, (r + 1) * per)
            mine.update({a[0][0]: a for a in follow(at, lambda q: q < stop)[1]})
        if mine != {s: a for s, a in truth.items() if s // per == r}:
            problems.append(("path", r))

    pieces = [((0, 0, 0), 0, min(step, total))]
    for s, ((_, h, j0), blocks) in truth.items():
        for j in range(j0, SPREAD_CHECKS):
            if key[s, h, j] is not None:
                stop = min(s * bits + (j + 2) * step, total) if j < SPREAD_CHECKS - 1 else end["end", s, h]
                pieces.append((state[s, h, j][:3], blocks + count[s, h, j], stop))
    for i, (s, h, p, b, k, blocks) in enumerate(extras):
        if s in truth and truth[s][0][1] == h:
            pieces.append(((p, b, k), truth[s][1] + blocks, end["extra", i]))
    stored = []
    for (p, b, k), g, stop in pieces:
        if p < stop and g < stream.total_blocks and int((stream.block_ends < p).sum()) != g:
            problems.append(("piece block number", p, g))
        while p < stop and g < stream.total_blocks:
            stored.append(p)
            taken, _, advance = symbol(p, b, k)
            p, k = p + taken, k + advance
            if k >= 64:
                k, b, g = 0, (b + 1) % H, g + 1
    if sorted(stored) != stream.starts:
        problems.append(("symbols stored", len(stored), len(set(stored)), len(stream.starts)))
    return {"bytes": stream.clean_bytes, "blocks": C, "segment": seg, "segments": nseg, "noted": noted, "pieces": len(pieces),
            "path": len(truth), "problems": problems}

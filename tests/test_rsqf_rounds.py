"""The rounds of an RSQF build's exact replay: a group of blocks whose spill
crosses into a group that is itself replayed is joined with it and replayed
again, and the second replay must not build on what the first left behind.
The rounds are modelled on the CPU over the oracle's sequential insert, and the
engine's blocks and return slots are compared with it on the GPU."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev

Q = 10
# Fingerprints by quotient (xN: N copies; remainder 0), two clusters each with
# offsets above 62 that touch: in the first set block 8 goes wrong when the
# joined group keeps the second one's earlier blocks, in the second set return
# slots do too.
SETS = {
    "blocks": (
    "130x4 131x2 132x7 133 134x7 135x2 136x7 137 138x3 139x2 140x9 141x9 142x4 143x6 144x4 145x5 146x5 147x5 "
    "148x2 149x2 150x3 151x5 152x7 153x6 154x6 155x3 156x4 157x4 158x6 159x6 160x8 161x6 162x8 163x4 164x4 165x8 "
    "166x6 167x4 168x5 322x4 323x2 324 325x2 326x3 327 328 329x3 330x3 331x4 332x2 333x2 334 335x3 336x5 338x2 "
    "339 351x2 352x2 353x2 354x2 355x5 357x2 358x4 359x4 360 361x3 362x4 363x3 364 365x5 366x3 367 368 369 370 "
    "371x2 372 373x6 375x7 376x3 377x4 378x2 379x4 380x2 381x5 382x2 384 387x3 390x2 393 396 397x2 401x2 402 403 "
    "404 406 407 409 410 411 413 419 421 422 427 433 437 440 441 442 446 449 451 452 453x2 455 457x2 458 460x2 "
    "461 463 464 465 466 469x2 473x3 474x2 477x2 485 494 496x2 497 500 501x2 502 504 527 "
    ),
    "slots": (
    "51x6 52x7 53x5 54x7 55x5 56x2 57x7 58x6 59x6 61x4 62 63x2 64x3 65x8 66x5 67x2 68x7 69x8 71x6 72x6 73x7 75x2 "
    "78x8 79x8 80x3 81x4 82x2 83x4 84x6 85x4 86x2 87x8 89x3 90x2 93x4 94x7 95x6 96x3 97x2 98x2 99 100x8 101x4 "
    "102x5 103x5 104x8 105x6 108x6 109x4 110x5 112x4 117 124 132 134 144 148 162 164 185 198 201 206 257 258 263 "
    "278 283 293 297 307 324x2 325x2 326x8 327 328x3 329x6 330 331x5 332x6 333x2 334x3 335x3 336x3 337x7 338x5 "
    "339x2 340x2 341 342 343 344x7 345x6 346 347x2 348x7 349x5 351x4 352x7 353x4 355x8 356x7 358x6 359x7 360x3 "
    "361x8 362x5 363 364x8 365x4 366x2 367x2 368x3 369x8 371x2 372x3 373x4 374x7 375 376x8 392 402 413 416 424 "
    "429 432 447 457 470 475 478 495 508 516 520 521 531 560 566x7 567 569x5 570x4 571x5 572x5 573x8 574x9 575x6 "
    "576x4 577x8 578x10 579x2 580x9 581x4 582x2 583 584x4 585x7 587x4 588x7 589x10 590x10 591x3 592x10 594 595x7 "
    "596x2 597x10 598x6 599x2 600x2 601x2 603x2 604 605x2 606x10 607x5 608x7 609x2 610x2 611x3 612 613x7 614x2 "
    "615x3 616x2 617x10 618x5 619x7 621 622x2 623x2 624x4 625x2 627x9 628x2 629 646 648 659 665 667 673 674 675 "
    "702 710 730 739 768 776 782 789 790 822 827 833 835 "
    ),
}


def fingerprints(name, rbits):
    fps = []
    for w in "".join(SETS[name]).split():
        quotient, _, copies = w.partition("x")
        fps += [int(quotient) << rbits] * int(copies or 1)
    return np.array(fps, np.uint32)


def bursts(seed, rbits):
    """Heavy bursts, each followed by about as much room as it spills."""
    rng = np.random.default_rng(seed)
    fps, x, room = [], int(rng.integers(0, 200)), (1 << Q) - 320
    while x < (1 << Q) and len(fps) < room:
        n0, length = len(fps), int(rng.integers(20, 90))
        copies = rng.integers(0, 2 * int(rng.integers(2, 7)), length)
        for k in range(min(length, (1 << Q) - x)):
            fps += [((x + k) << rbits) | int(rng.integers(0, 1 << rbits)) for _ in range(copies[k])]
        spill = max(len(fps) - n0 - length, 0)
        x += length + int(spill * rng.uniform(0.8, 1.3)) + int(rng.integers(0, 3) == 0) * 100
    fps = fps[:room]
    return np.sort(np.array([f for f in fps if (f >> rbits) < (1 << Q)], np.uint32))


class Model:
    """A sorted batch into an empty filter: canonical blocks, then every group
    (a run of blocks from one of offset 0) that holds an offset above 62 is
    replayed with the sequential insert, joined with its successor when it
    writes past its end, until none does."""

    def __init__(self, fps, rbits):
        self.fps, self.rbits, self.bb = fps, rbits, 17 + 8 * rbits
        self.nbl = O.rsqf_num_blocks(Q)
        qs = (fps >> rbits).astype(np.int64)
        i = np.arange(fps.size)
        self.pos = i + np.maximum.accumulate(qs - i)
        blocks = 64 * np.arange(self.nbl + 1)
        self.fhome, self.fpos = np.searchsorted(qs, blocks), np.searchsorted(self.pos, blocks)
        self.off = self.fhome - self.fpos
        self.home = qs // 64

    def canonical(self, upto):
        t = O.rsqf_new(Q, self.rbits)
        assert O.rsqf_layout_sorted(t, Q, self.fps[:upto], self.rbits) == 0
        return t

    def replay(self, t, ret, b, e, first):
        """One group; False: it wrote past block e."""
        bb, i0, i1 = self.bb, int(self.fhome[b]), int(self.fhome[min(e, self.nbl)])
        sus = [x for x in range(b, min(e, self.nbl)) if self.off[x] > 62]
        i = min(max(int(self.fpos[sus[0]]), i0), i1) if sus else i0
        if i >= i1:
            return True
        w, end = max(b, int(self.home[i])), e
        s = self.canonical(i)
        s[: w * bb] = 0
        hcur = self.home[i]
        while i < i1:
            h = int(self.home[i])
            if first and h > hcur and i == self.fhome[h]:
                hcur = h
                if np.array_equal(s[h * bb:], self.canonical(i)[h * bb:]):  # canonical again
                    later = [x for x in sus if x >= h]
                    i2 = min(max(int(self.fpos[later[0]]), i), i1) if later else i1
                    if i2 == i1:
                        end = h
                        break
                    if i2 > i:
                        s[h * bb:] = self.canonical(i2)[h * bb:]
                        i, hcur = i2, self.home[i2]
                        continue
            ret[i] = O.lib().or_rsqf_insert_fp(s, Q, self.rbits, int(self.fps[i]))
            if s[e * bb:].any():
                return False
            i += 1
        t[w * bb:end * bb] = s[w * bb:end * bb]
        return True

    def run(self):
        t, ret = self.canonical(self.fps.size), self.pos.astype(np.int32)
        start = [bool(o == 0) for o in self.off[:-1]] + [True]
        active = {max(x for x in range(B + 1) if start[x]) for B in range(self.nbl) if self.off[B] > 62}
        rounds = 0
        while active:
            crossed = []
            for b in sorted(active):
                e = next(x for x in range(b + 1, self.nbl + 2) if x > self.nbl or start[x])
                if not self.replay(t, ret, b, e, rounds == 0):
                    crossed.append((b, e))
            for _, e in crossed:
                if e <= self.nbl:
                    start[e] = False
            active = {max(x for x in range(b + 1) if start[x]) for b, _ in crossed}
            rounds += 1
        return t, ret, rounds


def sequential(fps, rbits):
    t = O.rsqf_new(Q, rbits)
    return t, np.array([O.lib().or_rsqf_insert_fp(t, Q, rbits, int(f)) for f in fps], np.int32)


@pytest.mark.parametrize("rbits", [5, 8])
def test_replay_rounds_model(oracle_lib, rbits):
    batches = [fingerprints(name, rbits) for name in SETS] + [bursts(s, rbits) for s in range(150)]
    joined = 0
    for fps in batches:
        if not fps.size or Model(fps, rbits).pos[-1] >= O.rsqf_num_blocks(Q) * 64:
            continue
        t, ret, rounds = Model(fps, rbits).run()
        want, slots = sequential(fps, rbits)
        assert np.array_equal(t, want) and np.array_equal(ret, slots)
        joined += rounds > 1
    assert joined >= 2


def keys_of(fps, rbits):
    """Keys with these fingerprints."""
    cand = O.mt_keys(1, 1 << 22)
    h = O.aphash(cand, Q, rbits)
    order = np.argsort(h, kind="stable")
    at = np.searchsorted(h[order], fps)
    assert np.array_equal(h[order][at], fps)
    return cand[order][at]


@pytest.mark.gpu
@pytest.mark.parametrize("rbits", [5, 8])
@pytest.mark.parametrize("which", list(SETS) + list(range(1, 10)))
def test_crossing_into_a_replayed_group(gqf, cuda, which, rbits):
    fps = bursts(which, rbits) if isinstance(which, int) else fingerprints(which, rbits)
    keys = keys_of(fps, rbits)
    o = O.rsqf_new(Q, rbits)
    want = O.rsqf_insert_sorted(o, Q, keys, rbits)
    f = gqf.initCQFGPU(Q, rbits)
    try:
        ret = cuda.empty(keys.size, dtype=cuda.int32, device="cuda")
        gqf.insertGPU(f, keys.size, to_dev(cuda, keys), ret)
        raw = gqf.rsqf_blocks_bytes(f)
        d = np.nonzero(raw != o)[0]
        assert d.size == 0, "%d bytes differ, first in block %d" % (d.size, d[0] // (17 + 8 * rbits))
        assert np.array_equal(ret.cpu().numpy(), want)
    finally:
        gqf.freeCQFGPU(f)

"""A standard filter's contents as a sorted fingerprint multiset, its table by
the oracle's canonical layout: what a sequence of operations leaves, in time
that does not grow with the clusters (the oracle's sequential operations are
compared with this layout in test_oracle.py)."""
import numpy as np

import oracle as O


class Contents:
    def __init__(self, q, r, keys, nodup):
        self.q, self.r = q, r
        f = self.fps(keys)
        self.f = np.unique(f) if nodup else np.sort(f)

    def fps(self, keys):
        return O.aphash(keys, self.q, self.r)

    def insert(self, keys):
        """Fingerprints not stored yet, once."""
        self.f = np.sort(np.concatenate([self.f, np.setdiff1d(self.fps(keys), self.f)]))

    def delete(self, keys):
        """One stored copy per occurrence."""
        want, times = np.unique(self.fps(keys), return_counts=True)
        first = np.searchsorted(self.f, want)
        have = np.searchsorted(self.f, want, side="right") - first
        drop = np.minimum(times, have)
        keep = np.ones(self.f.size, bool)
        at = np.repeat(first, drop) + np.arange(drop.sum()) - np.repeat(np.cumsum(drop) - drop, drop)
        keep[at] = False
        self.f = self.f[keep]

    def merge(self, other, nodup):
        f = np.concatenate([self.f, other])
        self.f = np.unique(f) if nodup else np.sort(f)

    def table(self):
        """The table, or None when the contents do not fit."""
        t = O.sqf_new(self.q, self.r)
        return t if O.sqf_layout_sorted(t, self.q, self.r, self.f) == 0 else None


def check(G, f, want, what=""):
    raw = G.table_bytes(f)
    if not np.array_equal(raw, want):
        d = np.nonzero(raw != want)[0]
        raise AssertionError("%s: %d bytes differ, first at %d" % (what, d.size, d[0]))

"""What the drift kernels' tables hold for a set of footpoints, counted from the
footpoints themselves (numpy): the tests use it to assert that a case reaches
the kinds of trips, cells and chunks it is meant to cover."""

import numpy as np

TRIP, CHUNK, LEFT, STAGED = 8, 16, 8, 48  # rows, rows, columns, columns


def drift_tables(fp, chain, nr, nu, nj):
    """far: cells whose taps leave their strip's staged columns; regular, empty:
    the trips (8 rows of a strip) of those kinds, and others the rest;
    empty_chunks: chunks (16 rows of 32 columns) without a cell in the box."""
    shape = (nj, nu, nr)
    rI, uI = fp["rI"].reshape(shape), fp["uI"].reshape(shape)
    chain = chain.reshape(shape)
    zero = (fp["out"].reshape(shape) != 0) & ~chain
    gather = ~zero & ~chain
    ns = nr // 32 if nr % 32 == 1 and nr > 32 else -(-nr // 32)
    wc = rI - (32 * np.minimum(np.arange(nr) // 32, ns - 1) - LEFT)
    inside = gather & (wc >= 0) & (wc <= STAGED - 4)
    nt = -(-nu // TRIP)
    regular, empty = np.zeros((nj, ns, nt), bool), np.zeros((nj, ns, nt), bool)
    for s in range(ns):
        cols = np.minimum(32 * s + np.arange(32), nr - 1)
        for t in range(nt):
            rows = slice(TRIP * t, TRIP * (t + 1))
            i, r, u = (a[:, rows][:, :, cols] for a in (inside, rI, uI))
            empty[:, s, t] = zero[:, rows][:, :, cols].all((1, 2))
            if i.shape[1] == TRIP:
                regular[:, s, t] = (i.all((1, 2)) & (np.diff(r, axis=1) == 0).all((1, 2)) &
                                    (np.diff(u, axis=1) == 1).all((1, 2)))
    sw, nc = -(-nr // 32), -(-nu // CHUNK)
    chunks = np.zeros((nj, sw, nc), bool)
    for s in range(sw):
        for c in range(nc):
            chunks[:, s, c] = zero[:, CHUNK * c:CHUNK * (c + 1), 32 * s:32 * s + 32].all((1, 2))
    return {"far": gather & ~inside, "regular": regular, "empty": empty,
            "others": ~regular & ~empty, "empty_chunks": chunks}

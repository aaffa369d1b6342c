"""SolverMatrix tables of hand-made block patterns, for shapes that a grid's nested
dissection does not give: cblks of any width, chains, arrowheads.  No PaStiX library."""
import numpy as np

from pastix_b200.refhost import BCSC, SolverStructure

FACTO_ID = {"potrf": 0, "sytrf": 1, "getrf": 2}


def block_structure(widths, faces, facto):
    """cblk k has widths[k] columns and, below its diagonal block, all the rows of the
    cblks faces[k] (ascending, later than k; the caller's pattern is closed under
    elimination).  Identity ordering."""
    w = np.asarray(widths, dtype=np.int64)
    cn = w.size
    first = np.concatenate([[0], np.cumsum(w)])
    n = int(first[-1])
    nblk = np.array([1 + len(f) for f in faces], dtype=np.int64)
    fblok = np.concatenate([[0], np.cumsum(nblk)])
    bf = np.array([b for k in range(cn) for b in (k, *faces[k])], dtype=np.int64)
    bown = np.repeat(np.arange(cn), nblk)
    rows = w[bf]
    roff = np.cumsum(rows) - rows
    roff -= roff[fblok[bown]]
    stride = np.add.reduceat(rows, fblok[:-1])
    off = bf != bown
    brow = np.nonzero(off)[0]
    brow = brow[np.argsort(bf[brow], kind="stable")]
    brownum = np.concatenate([[0], np.cumsum(np.bincount(bf[off], minlength=cn))])
    browind = np.full(bf.size + 1, -1)
    browind[brow] = np.arange(brow.size)
    app = lambda a, v: np.ascontiguousarray(np.concatenate([a, [v]]), dtype=np.int64)  # noqa: E731
    return SolverStructure(
        n, cn, int(bf.size), int(brow.size), int((stride * w).sum()), FACTO_ID[facto], app(first[:-1], n),
        app(first[1:] - 1, n), fblok.astype(np.int64), app(stride, 0), app(first[:-1], n), brownum.astype(np.int64),
        brownum.astype(np.int64), np.zeros(cn + 1, np.int32), app(first[bf], n), app(first[bf] + rows - 1, n),
        app(bown, cn + 1), app(bf, cn + 1), app(roff * w[bown], 0), browind.astype(np.int64), brow.astype(np.int64),
        np.arange(n), np.arange(n), 0.0, cn)


def dense_structure(widths, facto):
    return block_structure(widths, [list(range(k + 1, len(widths))) for k in range(len(widths))], facto)


def chain_structure(widths, facto):
    return block_structure(widths, [[k + 1] if k + 1 < len(widths) else [] for k in range(len(widths))], facto)


def bcsc_of(A, facto):
    """bcsc of a SciPy sparse matrix with a symmetric pattern (identity ordering)."""
    A = A.tocsc()
    A.sort_indices()
    U = None
    if facto == "getrf":
        T = A.T.tocsc()
        T.sort_indices()
        U = T.data
    return BCSC(A.shape[0], A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data, U,
                float(np.sqrt((A.data ** 2).sum())))

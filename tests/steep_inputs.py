"""Initial conditions with deep one-sided trees, and a replay on the CPU of the
order in which the aggregation's second kernel (rise_kernel in k_tree.cu)
takes the finished subtrees of each 256-particle run."""
import numpy as np

RUN = 256    # particles of a run
LANES = 32   # subtrees of a run taken at once, one a lane


def _stars(gcs, xyz, seed):
    st = np.zeros(len(xyz), gcs.STAR_DTYPE)
    rng = np.random.default_rng(seed)
    for k, f in enumerate(("x", "y", "z")):
        st[f] = xyz[:, k]
        st["v" + f] = rng.normal(0, 1e-3, len(xyz))
    st["mass"] = rng.uniform(0.5, 1.5, len(xyz))
    return st


def corner_chain(gcs, n_core=2348, mirror=False):
    """Coincident particles in one corner of the Morton cube and one at every
    power of two along each axis: one node of the chain a level."""
    top = 2097151.0
    out = [(0.0, 0.0, 0.0)] * n_core + [(top, 0.0, 0.0)]
    for k in range(21):
        for axis in range(3):
            p = [0.0, 0.0, 0.0]
            p[axis] = float(1 << k)
            out.append(tuple(p))
    xyz = np.array(out)
    return _stars(gcs, top - xyz if mirror else xyz, 1)


def steep_profile(gcs, n_core=5000, n_outer=1200, seed=0):
    """A dense core and particles of log-uniform radius around it, in the
    middle of a symmetric box."""
    rng = np.random.default_rng(seed)
    core = rng.normal(0, 1e-6, (n_core, 3))
    d = rng.normal(0, 1, (n_outer, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    outer = d * np.exp(rng.uniform(np.log(1e-6), 0.0, n_outer))[:, None]
    box = np.array([[-1.0, -1.0, -1.0], [1.0, 1.0, 1.0]])
    return _stars(gcs, np.concatenate([core, outer, box]), seed)


def sorted_tree(oracle, stars):
    xyz = np.stack([stars[f] for f in ("x", "y", "z", "mass")], 1).astype(np.float32)
    lo, hi = oracle.bounds(xyz)
    return oracle.build(oracle.sort(oracle.encode(xyz, lo, hi))[0])


def subtrees(tree, n):
    """For each run: (first particle, subtree, climb step at which it was
    finished) of every finished subtree whose parent is above the run, by first
    particle.  Subtrees >= n - 1 are particles."""
    cl, cr, re, par, lp = (a.astype(np.int64) for a in tree)
    own = np.arange(n - 1)
    lo, hi = np.minimum(own, re), np.maximum(own, re)
    local = lo // RUN == hi // RUN
    step = np.zeros(2 * n - 1, np.int64)  # particles: 0
    for k in np.argsort(hi - lo, kind="stable"):  # children before parents
        step[k] = 1 + max(step[c] if c < n - 1 else 0 for c in (cl[k], cr[k]))
    out = [[] for _ in range((n + RUN - 1) // RUN)]
    for k in range(n - 1):
        if not local[k]:
            for c in (cl[k], cr[k]):
                first = c - (n - 1) if c >= n - 1 else lo[c]
                if c >= n - 1 or local[c]:
                    out[first // RUN].append((int(first), int(c), int(step[c]) if c < n - 1 else 0))
    return [sorted(r) for r in out]


def by_position(run):
    return [c for _, c, _ in run]


def by_completion(run):
    return [c for _, c, _ in sorted(run, key=lambda s: (s[2], s[0]))]


def replay(tree, n, order):
    """Take every run's subtrees in the given order, lane l the entries l,
    l + 32, ... one after another: a left child hands over and stops, a right
    child waits for its left one, then goes on from their parent.  Returns the
    number of lanes that never finish."""
    cl, cr, _, par, lp = (a.astype(np.int64) for a in tree)
    up = lambda c: int(lp[c - (n - 1)] if c >= n - 1 else par[c])  # noqa: E731
    lanes = []
    for run in subtrees(tree, n):
        todo = order(run)
        lanes += [todo[i::LANES] for i in range(min(LANES, len(todo)))]
    handed = set()
    moved = True
    while moved:
        moved = False
        for todo in lanes:
            while todo:
                c, p = todo[0], up(todo[0])
                if p < 0 or cl[p] == c:
                    if p >= 0:
                        handed.add(p)
                    todo.pop(0)
                elif p in handed:
                    todo[0] = p
                else:
                    break
                moved = True
    return sum(1 for todo in lanes if todo)

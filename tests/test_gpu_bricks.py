"""The builds through bricks (16^3 of a dense grid, 8^3 of a mesh fold): one
brick as the root, ragged and misaligned grids, cache blocks of a brick's size,
far pointers right above the bricks, and cubes whose brick codes are too many
for the dense level arrays.  Words bit-exact to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def budget(oracle, shape, edge):
    """A budget whose cache blocks have this edge (None: one block)."""
    mem = 3000
    while edge is not None and oracle.cache_block(shape[2], shape[1], shape[0], mem) < edge:
        mem += mem // 16
    return 1 << 30 if edge is None else mem


@pytest.mark.parametrize("shape,density,edge", [
    ((16, 16, 16), 1.0, None),      # the brick is the root
    ((16, 16, 16), 0.01, None),
    ((15, 13, 16), 0.4, None),      # odd depth: the last slice is dropped
    ((32, 32, 32), 0.0, None),
    ((64, 64, 64), 1.0, None),      # every offset above a brick is far
    ((17, 33, 65), 0.3, None),      # rows off the 16-byte boundary
    ((50, 47, 100), 0.002, None),   # partial bricks in every direction
    ((33, 40, 48), 0.1, 16),        # 16^3 cache blocks
    ((65, 64, 40), 0.05, 32),       # 32^3 cache blocks
    ((9, 20, 2100), 0.2, None),     # 4096^3 cube: compacted nodes
    ((35, 36, 2052), 0.1, 64),      # the same with cache blocks
    ((35, 36, 2052), 0.1, 128),
])
def test_dense_builds(svo, oracle, scenes, shape, density, edge):
    mem = budget(oracle, shape, edge)
    g = scenes.random_grid(shape, density, sum(shape))
    if edge is not None:
        # a cache block whose only voxels lie in the dropped slice
        assert oracle.cache_block(shape[2], shape[1], shape[0], mem) == edge
        z = (shape[0] - 1) // edge * edge
        g[z:, :edge, :edge] = 0
        g[shape[0] - 1, 3, 5] = 77
    ow, oc = oracle.build_dense(g, mem)
    tree = svo.VoxelOctree(svo.VoxelData(g, mem))
    assert np.array_equal(tree.words(), ow)
    assert np.array_equal(tree.center(), oc)


@pytest.mark.parametrize("shape,offset", [
    ((9, 20, 2101), 0),    # rows off the 16-byte boundary
    ((70, 20, 2050), 0),
    ((20, 2101, 40), 1),   # whole rows, the first off it
    ((2101, 36, 17), 3),
])
def test_unaligned_rows_in_large_cubes(cuda, svo, oracle, scenes, shape, offset):
    """4096^3 cubes, in which a CTA visits sixteen bricks and those inside the
    grid have padding between them, read a word at a time: the bits of one
    brick while the next one's are formed."""
    torch = cuda
    g = scenes.random_grid(shape, 0.3, sum(shape))
    flat = torch.zeros(g.size + offset, dtype=torch.int32, device="cuda")
    dev = flat[offset:].view(shape)
    dev.copy_(torch.from_numpy(g.view(np.int32)))
    ow, oc = oracle.build_dense(g)
    for _ in range(3):
        tree = svo.VoxelOctree(svo.VoxelData(dev, 1 << 30))
        assert np.array_equal(tree.words(), ow)
        assert np.array_equal(tree.center(), oc)


@pytest.mark.parametrize("side,thin,threads,mem", [
    (8, 1.0, 2, 1 << 30),         # one 8^3 brick
    (60, 0.5, 5, 1 << 30),
    (700, 0.03, 16, 1 << 30),     # 1024^3 cube, a needle
    (1500, 0.015, 16, 1 << 30),   # 2048^3 cube: compacted nodes
    (1500, 0.015, 4, 3 << 20),    # the same in small cache blocks
])
def test_mesh_builds(svo, oracle, scenes, side, thin, threads, mem):
    pos, faces, col = scenes.displaced_icosphere(3, side)
    pos = pos * np.array([1.0, thin, thin], np.float32)
    col = col.astype(np.float32)
    tree = svo.VoxelOctree(svo.VoxelData(svo.PlyLoader.from_arrays(pos, faces, colors=col), side, mem, threads))
    ow, oc = oracle.build_mesh(pos, faces, side, threads, mem, colors=col)
    assert np.array_equal(tree.words(), ow)
    assert np.array_equal(tree.center(), oc)


def _fan(n, rng):
    """n small triangles in one corner of the unit cube, and one across it."""
    at = rng.uniform(0.1, 0.104, (n, 1, 3))
    pos = np.concatenate([(at + rng.uniform(-0.004, 0.004, (n, 3, 3))).reshape(-1, 3),
                          [[0.0, 0.0, 0.0], [1.0, 0.2, 0.9], [0.9, 1.0, 0.1]]]).astype(np.float32)
    return pos, np.arange(3 * (n + 1), dtype=np.int32).reshape(-1, 3)


@pytest.mark.parametrize("side,n,threads,mem", [
    (64, 40, 4, 1 << 30), (64, 480, 4, 1 << 30),    # one brick holds tens, hundreds of triangles
    (64, 900, 4, 1 << 30), (64, 4000, 4, 1 << 30),  # thousands, a CTA's sort
    (64, 4600, 4, 1 << 30),                         # and more than that sorts
    (16, 30, 512, 1 << 30), (40, 60, 4096, 1 << 30),  # sub-blocks inside a brick: several pairs of one triangle
    (40, 60, 512, 5 * 16 ** 3 + 3000),              # and several cache blocks
    (16, 600, 4, 1 << 30), (16, 3001, 512, 1 << 30),  # hundreds of pairs in every brick: rounds of 16
    (1027, 50, 8, 1 << 30),                         # beyond the table of brick codes
])
def test_mesh_pairs_by_brick(svo, oracle, monkeypatch, side, n, threads, mem):
    """Pairs laid out through the table of brick codes, and sorted: the words
    of the block-after-block fold, and of the oracle."""
    rng = np.random.default_rng(side + n)
    pos, faces = _fan(n, rng)
    col = rng.uniform(0, 1, pos.shape).astype(np.float32)
    got = svo.VoxelOctree(svo.VoxelData(svo.PlyLoader.from_arrays(pos, faces, colors=col), side, mem, threads)).words()
    monkeypatch.setenv("SVO_MESH_BLOCK_BUFFER", "1")
    want = svo.VoxelOctree(svo.VoxelData(svo.PlyLoader.from_arrays(pos, faces, colors=col), side, mem, threads)).words()
    assert np.array_equal(got, want)
    if side <= 64:
        ow, _ = oracle.build_mesh(pos, faces, side, threads, mem, colors=col)
        assert np.array_equal(got, ow)


@pytest.mark.parametrize("n", [4096, 1 << 19])
@pytest.mark.parametrize("threads", [1, 16])
def test_more_pairs_than_can_be_laid_out(svo, n, threads):
    """Triangles across a 1024^3 cube in sub-blocks of all or a sixteenth of
    it, 2^31 to 2^40 (brick, triangle) pairs: refused, after a count that
    leaves the table of bricks in range, and the next build is right."""
    pos = np.array([[0, 0, 0], [1, 1, 0.1], [0.2, 0.9, 1]], np.float32)
    mem = 8 << 30  # one cache block

    def build(k):
        loader = svo.PlyLoader.from_arrays(pos, np.tile(np.arange(3, dtype=np.int32), (k, 1)))
        return svo.VoxelOctree(svo.VoxelData(loader, 1024, mem, threads))

    with pytest.raises(svo.SvoError) as e:
        build(n)
    assert e.value.code == svo.SVO_ERR_LIMIT
    assert build(1).num_words() > 100_000


@pytest.mark.parametrize("n_threads", [1, 24])
def test_builds_side_by_side(svo, oracle, scenes, n_threads):
    """More builds, tables and mesh builds at a time than there are page-locked
    report slots: the rest report through copies."""
    import threading
    grid = scenes.sphere_scene(64, 9, 3)
    want, _ = oracle.build_dense(grid)
    pos, faces, col = scenes.displaced_icosphere(2, 5)
    mw, _ = oracle.build_mesh(pos, faces, 40, 4, 1 << 30, colors=col.astype(np.float32))
    entries = svo.VoxelOctree.from_words(want, np.full(3, 0.5, np.float32)).table_size()
    go, bad = threading.Barrier(n_threads), []

    def work():
        go.wait()
        for _ in range(6):
            t = svo.VoxelOctree(svo.VoxelData(grid, 1 << 30))
            if not (np.array_equal(t.words(), want) and t.table_size() == entries):
                bad.append("dense")
            m = svo.VoxelOctree(svo.VoxelData(svo.PlyLoader.from_arrays(pos, faces, colors=col.astype(np.float32)), 40,
                                              1 << 30, 4))
            if not np.array_equal(m.words(), mw):
                bad.append("mesh")

    ts = [threading.Thread(target=work) for _ in range(n_threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad

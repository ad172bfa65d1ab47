"""The viewer traces one octree from 16 host threads at once, each thread
calling VoxelOctree::raymarch for its own pixels (Main.cpp:342-367).  The
host-buffer calls that replace it are made the same way here: 16 threads on
two freshly built octrees (so the first calls race to build the descriptor
table), mixing svo_trace_host, svo_trace_image_host and single-ray
raymarch, and every result is the oracle's, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_THREADS = 16
W, H = 96, 64


def _check(res, ref, what):
    assert np.array_equal(res["hit"], ref["hit"]), what
    assert np.array_equal(res["t"].view(np.uint32), ref["t"].view(np.uint32)), what
    assert np.array_equal(res["word"], ref["word"]), what
    assert np.array_equal(res["rgb"][:, 0].view(np.uint32), ref["grey"].view(np.uint32)), what


def test_host_calls_from_16_threads(svo, oracle, scenes):
    grids = [scenes.sphere_scene(128, 20, 5), scenes.terrain_scene(128, 20, 6)]
    built = [oracle.build_dense(g) for g in grids]
    trees = [svo.VoxelOctree(svo.VoxelData(g)) for g in grids]
    cams = [scenes.orbit_cameras(N_THREADS, 3 + k, built[k][1]) for k in range(2)]
    jobs = []
    for i in range(N_THREADS):
        k = i % 2
        cam = cams[k][i]
        jobs.append((k, scenes.camera_rays(cam, W, H), scenes.headlight(cam)))
    results = [None] * N_THREADS
    singles = [None] * N_THREADS
    errors = []
    start = threading.Barrier(N_THREADS)

    def work(i):
        try:
            k, rays, light = jobs[i]
            start.wait()
            for rep in range(3):
                if (i + rep) % 2:
                    r = trees[k].trace_host(rays, light=light, outputs=("hit", "t", "word", "rgb"))
                else:
                    r = trees[k].trace_image_host(rays, W, H, light=light, outputs=("hit", "t", "word", "rgb"))
                if rep == 0:
                    results[i] = r
                else:
                    for key in r:
                        if not np.array_equal(r[key], results[i][key]):
                            raise AssertionError("thread %d call %d differs in %s" % (i, rep, key))
            # the reference's own call shape: one ray per call
            singles[i] = [trees[k].raymarch(rays[j, :3], rays[j, 3:]) for j in range(0, rays.shape[0], 97)]
        except Exception as e:  # re-raised on the main thread
            errors.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(N_THREADS)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=600)
    assert not any(t.is_alive() for t in threads)
    assert not errors, errors
    hits = 0
    for i, (k, rays, light) in enumerate(jobs):
        ref = oracle.raymarch(built[k][0], rays, light=light)
        _check(results[i], ref, "thread %d" % i)
        hits += int((ref["hit"] == 1).sum())
        for n, j in enumerate(range(0, rays.shape[0], 97)):
            hit, word, t = singles[i][n]
            assert hit == (ref["hit"][j] != 0), (i, j)
            if ref["hit"][j] == 1:
                assert word == int(ref["word"][j]) and np.float32(t) == ref["t"][j], (i, j)
    assert hits > N_THREADS * 500


@pytest.mark.parametrize("mode,own_thread", [("thread_local", False), ("relaxed", False), ("relaxed", True)])
def test_destroy_beside_a_capture(cuda, svo, scenes, mode, own_thread):
    """An octree destroyed while another call is being captured: the capture
    goes on, and the octree's memory goes back only once the device is idle."""
    torch = cuda
    tree = svo.VoxelOctree(svo.VoxelData(scenes.sphere_scene(64, 9, 3)))
    other = svo.VoxelOctree(svo.VoxelData(scenes.sphere_scene(64, 9, 4)))
    rays = torch.from_numpy(scenes.random_rays(4096, 5)).cuda()
    out = {"t": torch.zeros(4096, device="cuda")}
    tree.trace(rays, out=out)
    torch.cuda.synchronize()
    want = out["t"].clone()
    assert bool(torch.isfinite(want).any())
    busy, ended, idle = torch.cuda.Stream(), torch.cuda.Event(), []

    def destroy():
        other.close()
        idle.append(ended.query())

    graph = torch.cuda.CUDAGraph()
    st = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=st, capture_error_mode=mode):
        tree.trace(rays, out=out, stream=st)
        with torch.cuda.stream(busy):
            torch.cuda._sleep(40_000_000)  # about 20 ms
            ended.record(busy)
        if own_thread:
            destroy()
        else:
            t = threading.Thread(target=destroy)
            t.start()
            t.join()
    assert idle == [True]
    out["t"].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out["t"], want)


def test_destroy_inside_a_global_capture(cuda, svo):
    """Where no wait is allowed the memory is kept aside: no later octree gets
    it, and svo_trim_memory returns it once the capture has ended."""
    import ctypes
    torch = cuda
    rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")
    grid = torch.ones((256, 256, 256), dtype=torch.int32, device="cuda")
    tree = svo.VoxelOctree(svo.VoxelData(grid))
    held, size = tree.device_words_ptr(), 4 * tree.num_words()
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    handle, graph = ctypes.c_void_p(st.cuda_stream), ctypes.c_void_p()
    assert rt.cudaStreamBeginCapture(handle, 0) == 0
    tree.close()
    assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) != 0  # as with any free in such a capture
    rt.cudaGetLastError()
    later = [svo.VoxelOctree(svo.VoxelData(grid)) for _ in range(2)]
    at = [t.device_words_ptr() for t in later]
    assert all(p + size <= held or held + size <= p for p in at)
    before = torch.cuda.mem_get_info()[0]
    svo.trim_memory()
    assert torch.cuda.mem_get_info()[0] - before >= size
    assert later[0].num_words() * 4 == size

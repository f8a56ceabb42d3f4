"""Chunk boundaries of the host-buffer trace pipeline (csrc/host_chunks.hpp):
on CPU, for every chunk size from the smallest up and the counts around each
rule's edges, the boundaries ascend from 0 to n; on the GPU, traces with small
RAY_HOST_CHUNK values give the hits of the unpiped call."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from raydemo_b200 import api, capi, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
#include "host_chunks.hpp"
#include <cstdio>
int main() {
    unsigned long long n, chunk;
    while (std::scanf("%llu %llu", &n, &chunk) == 2) {
        const std::vector<uint64_t> cut = rg::trace_cuts(n, chunk);
        uint64_t big = 0;
        bool ok = cut.front() == 0 && cut.back() == n;
        for (size_t k = 0; k + 1 < cut.size(); k++) {
            ok = ok && (cut[k] < cut[k + 1] || n == 0);
            big = std::max(big, cut[k + 1] - cut[k]);
        }
        std::printf("%llu %llu %d %zu %llu\\n", n, chunk, (int)ok, cut.size() - 1, (unsigned long long)big);
        std::fflush(stdout);
    }
}
"""


def test_cuts_ascend_for_every_chunk_size(tmp_path):
    src, exe = tmp_path / "cuts.cpp", str(tmp_path / "cuts")
    src.write_text(PROGRAM)
    subprocess.run([os.environ.get("CXX") or shutil.which("g++"), "-std=c++17", "-O1", f"-I{ROOT}/raydemo_b200/csrc", "-o", exe, str(src)],
                   check=True)
    pairs = [(n, max(n, 1)) for n in (0, 1, 5000, 1 << 20)]  # one chunk
    for chunk in (1024, 2048, 3072, 4096, 5120, 8192, 262144):
        edges = {chunk + 1, 2 * chunk, 4 * chunk - 4096, 4 * chunk, 6 * max(1024, chunk // 4), 9 * chunk}
        pairs += [(n, chunk) for e in edges for n in range(e - 2, e + 3) if n > chunk]
    pairs += [(n, c) for c in (1024, 2048) for n in range(c + 1, 8200, 7)]
    for n in (262145, 1048575, 1048576, 1048583, 4194304, 4194305, 0xFFFFFFFF):  # the default chunk
        c = max(262144, (n + 3) // 4 + 1023 & ~1023)
        pairs.append((n, c))
    out = subprocess.run([exe], input="".join(f"{n} {c}\n" for n, c in pairs), capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout.splitlines()[-1:]
    rows = [tuple(int(v) for v in l.split()) for l in out.stdout.splitlines()]
    assert len(rows) == len(pairs)
    for n, chunk, ok, parts, big in rows:
        assert ok, (n, chunk)
        assert big <= max(chunk, 2048, n if chunk >= n else 0), (n, chunk, big)
        assert parts <= n // chunk + 6, (n, chunk, parts)


@pytest.mark.gpu
@pytest.mark.parametrize("chunk", [1024, 2048])
def test_small_chunks_give_the_unpiped_hits(cuda_device, chunk, monkeypatch):
    import torch

    r = api.Renderer(16, 16)
    attrs, idx = scenes.triangle_soup_mesh(scenes.random_triangles(2000, seed=3, mean_edge=0.05))
    sc = r.CreateScene()
    m = sc.AddMaterial()
    sc.AddMeshInstance(sc.AddMesh(attrs, idx, [(m, 0, len(idx))]))
    rays = torch.from_numpy(scenes.incoherent_rays(70000, seed=4)).pin_memory()

    def trace(n, value):
        monkeypatch.setenv("RAY_HOST_CHUNK", str(value))
        hits = torch.full((n, 4), -7, dtype=torch.int32).pin_memory()
        obj = torch.full((n,), -7, dtype=torch.int32).pin_memory()
        capi.check(capi.lib().ray_scene_trace_closest(sc.handle, rays.data_ptr(), n, hits.data_ptr(), obj.data_ptr(), capi.RAY_MEM_HOST, None))
        return hits.numpy(), obj.numpy()

    for n in (1025, 3073, 4096, 4097, 5000, 6143, 6144, 6145, 12289, 70000):  # 70000: more chunks than work counters
        hits, obj = trace(n, chunk)
        want, want_obj = trace(n, 0)
        assert np.array_equal(hits, want) and np.array_equal(obj, want_obj), n

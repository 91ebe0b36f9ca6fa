"""The marching-cubes table against the rule the mesher's classification rests
on: a case's triangles use exactly the edges whose corners differ in sign."""
import os
import re


def test_triangles_use_the_edges_of_a_sign_change():
    src = os.path.join(os.path.dirname(__file__), "..", "merge_fusion_gb300", "csrc")
    words = [int(w, 16) for w in re.findall(r"0x([0-9a-f]{16})ull", open(os.path.join(src, "mc_table.cuh")).read())]
    mesh = open(os.path.join(src, "kifi_mesh.cu")).read()
    corners = int(re.search(r"kEdgeCorners = 0x([0-9a-f]+)ull", mesh).group(1), 16)
    axes = int(re.search(r"kEdgeAxes = 0x([0-9a-f]+)u", mesh).group(1), 16)
    assert len(words) == 256
    bit = [2, 3, 6, 7, 1, 0, 5, 4]  # the case bit of each corner
    for case, w in enumerate(words):
        used = {w >> (4 * t) & 15 for t in range(3 * (w >> 60))}
        neg = [case >> b & 1 for b in bit]
        differ = set()
        for e in range(12):
            c, a = corners >> (4 * e) & 15, axes >> (2 * e) & 3
            if neg[c] != neg[c | 1 << a]:
                differ.add(e)
        assert used == differ, case

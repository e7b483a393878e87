"""__ldg reads through the non-coherent cache, which is right only for data that
nobody writes while the reading kernel exists.  The raster and order kernels
start while the prepare kernel still writes the visible records, their order and
the model records, so every __ldg names a table that the host uploads.  (Read
from the source: on the device a stale line is a matter of luck.)"""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "habitat-sim_gb300", "csrc",
                      "kernels.cu")
# Vertices, indices, meshes; texels of a texture (base); normals; local transforms
# (load_matrix); the finished plane that a gather packs (from).
UPLOADED = re.compile(r"&p\.(pos|color|uv|indices|meshes)\[|base \+ |&vertex_normals\[|"
                      r"reinterpret_cast<const float4\*>\(m\)|reinterpret_cast<const uint4\*>\(from\)|from\)")


def test_every_non_coherent_load_reads_an_uploaded_table():
    text = open(SOURCE).read()
    code = re.sub(r"//[^\n]*", "", text)
    loads = [code[m.end():m.end() + 60] for m in re.finditer(r"__ldg\(", code)]
    assert len(loads) > 10
    assert [x for x in loads if not UPLOADED.match(x)] == []

"""Dynamic shared memory that a kernel reads in 16-byte words says so: without an
alignment its place behind the static part is up to the compiler."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepmd-jax_b200", "csrc")


def test_dynamic_shared_memory_is_aligned_where_it_is_read_in_vectors():
    bad = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            src = f.read()
        vectors = re.search(r"reinterpret_cast<(const )?(float4|int4|uint4) \*>", src)
        for m in re.finditer(r"extern __shared__ ([^;]*);", src):
            if vectors and not re.search(r"__align__\((16|128|1024)\)", m.group(1)):
                bad.append("%s:%d" % (name, src[:m.start()].count("\n") + 1))
    assert not bad

"""Kernels that are launched programmatically (they may start while the kernel before them still runs) must wait for it
on every way out: a grid that ends without waiting lets the kernel behind it, which only waits for that grid, run beside
the one in front.  Read from the sources: no GPU is needed, and no wait has to be made to run out."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "retrievalattention_b200", "csrc")
WAIT = re.compile(r"\bri_pdl_(?:wait|enter)\s*\(\s*\)")


def sources():
    files = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
    strip = lambda text: re.sub(r"/\*.*?\*/|//[^\n]*", "", text, flags=re.S)      # noqa: E731
    return [strip(open(f).read()) for f in files]


def kernel_bodies(text):
    """(name, body) of every kernel defined in a comment-free source."""
    for m in re.finditer(r"__global__\b[^;{]*?\b(\w+)\s*\((?=[^;{]*\{)", text):
        name = re.findall(r"(\w+)\s*\(", text[m.start():text.index("{", m.end())])
        name = [n for n in name if n.endswith("_kernel")][0]
        start = text.index("{", m.end())
        depth, i = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield name, text[start + 1:i - 1]


def unguarded_exits(body):
    """Returns in front of the kernel's unconditional wait that no wait in their own block precedes (with the wait itself
    missing: the kernel's end)."""
    blocks, bad, i = [[False]], [], 0           # per open block: whether a wait stands in it, so far
    while i < len(body):
        if body[i] == "{":
            blocks.append([False])
        elif body[i] == "}":
            blocks.pop()
        elif WAIT.match(body, i):
            blocks[-1][0] = True
            if len(blocks) == 1:
                return bad
        elif re.compile(r"\breturn\s*;").match(body, i) and not any(b[0] for b in blocks):
            bad.append(body[max(0, i - 60):i + 7].split("\n")[-1].strip())
        i += 1
    return bad + ["end of the kernel"]


def test_the_check_sees_a_missing_wait():
    early = "if (s_skip) return; ri_pdl_wait(); work();"
    assert unguarded_exits(early) == ["if (s_skip) return;"]
    assert unguarded_exits("if (s_skip) { ri_pdl_wait(); return; } ri_pdl_wait(); if (x) return; work();") == []
    assert unguarded_exits("if (a) { ri_pdl_wait(); } work();") == ["end of the kernel"]
    assert list(kernel_bodies("__global__ void __launch_bounds__(f(1), 1)\nmy_kernel(int a) { if (a) { b(); } }")) == \
        [("my_kernel", " if (a) { b(); } ")]


def test_programmatically_launched_kernels_wait_on_every_way_out():
    texts = sources()
    calls = r"(?:ri_launch_pdl_id\(\s*\w+|ri_launch_pdl_cluster\(\s*\w+,\s*\w+|cudaLaunchKernelEx\(\s*&\w+),\s*(?:\w+::)*(\w+_kernel)\b"
    bodies = {n: b for t in texts for n, b in kernel_bodies(t)}
    launched = {n for t in texts for n in re.findall(calls, t)} | {n for n, b in bodies.items() if "ri_pdl_" in b}
    assert {"kmeans_assign_wide_kernel", "kmeans_assign_resident_kernel", "kmeans_bucket_kernel", "kmeans_update_kernel",
            "dense_decode_kernel", "dense_combine_kernel", "dense_append_kernel", "rmsnorm_kernel"} <= launched
    found = {n: unguarded_exits(bodies[n]) for n in sorted(launched)}
    assert not any(found.values()), found


def test_every_programmatic_launch_asks_the_switch():
    """RI_PDL_MASK covers them all: the attribute is set in one place, behind the mask."""
    uses = [t for t in sources() if "cudaLaunchAttributeProgrammaticStreamSerialization" in t]
    assert len(uses) == 1 and uses[0].count("cudaLaunchAttributeProgrammaticStreamSerialization") == 1
    assert re.search(r"if \(\(ri_pdl_mask\(\) >> id\) & 1\) \{[^}]*cudaLaunchAttributeProgrammaticStreamSerialization", uses[0])

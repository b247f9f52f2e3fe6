"""Rules of the CUDA sources that the compiler does not check."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "miles_b200", "ops", "csrc")


def _closing(text, at, pair):
    """Index behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise ValueError(text[at:at + 80])


def _kernels(text):
    """(name, parameters, body) of every kernel that is defined in `text`."""
    for start in re.finditer(r"__global__\s+void\b", text):
        at = start.end()
        while True:
            word = re.compile(r"\s*(\w+)\s*\(").match(text, at)
            end = _closing(text, word.end() - 1, "()")
            if word.group(1) not in ("__launch_bounds__", "__cluster_dims__"):
                break
            at = end
        if (body := re.compile(r"\s*\{").match(text, end)):
            yield word.group(1), text[word.end():end - 1], text[body.end():_closing(text, body.end() - 1, "{}")]


# weights and constant tables: what writes them has finished when a kernel that was launched behind it starts
STATIC = {"w", "w13", "w2", "norm_w", "nw", "ls", "fw", "qw", "kw", "q_norm", "k_norm", "kv_norm", "lvec", "sink", "freq", "embed", "table"}


def test_kernels_that_wait_for_the_one_in_front_promise_nothing_about_what_it_writes():
    """A load through a `__restrict__` parameter may be moved up in front of the dependency wait (pdl.cuh)."""
    waiting = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        for name, parameters, body in _kernels(open(path).read()):
            if "pdl_wait" in body:
                waiting += 1
                for p in parameters.split(","):
                    assert "__restrict__" not in p or ("const" in p and p.split()[-1] in STATIC), (os.path.basename(path), name, p.strip())
    assert waiting > 50                                     # the sources were read
    for path in glob.glob(os.path.join(CSRC, "*.cu")):      # … and no step of the optimizer lets the next kernel start early
        for name, _, body in _kernels(open(path).read()):
            assert "adamw" not in name or "pdl_trigger" not in body

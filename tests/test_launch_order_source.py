"""Kernels that may start before the one before them is done (those that call
pdl(), jsd_common.cuh) must not promise the compiler that their data stays
unchanged from the kernel's first instruction on: a `__restrict__` kernel
parameter lets its loads move above the wait. Only tables that no kernel writes
may carry it. Reads the sources; no GPU."""
import glob
import os
import re

from conftest import REPO

TABLES = {"tw", "twtab", "vinv", "weights"}  # twiddles, V^-1, quadrature weights: written once, at plan creation


def _kernels():
    for path in sorted(glob.glob(os.path.join(REPO, "jax-spectral-dns_b200", "csrc", "*.cu*"))):
        src = open(path).read()
        for m in re.finditer(r"__global__\s+void", src):
            brace = src.index("{", m.start())
            depth, end = 0, brace
            while True:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
                if depth == 0:
                    break
            head, body = src[m.start():brace], src[brace:end]
            name = re.search(r"\b(k_\w+)\s*\((?=[^()]*\)\s*$)", head)
            yield name.group(1), head[name.end():], body  # name, parameters, body


def test_early_started_kernels_promise_nothing_about_their_data():
    early = [(name, head) for name, head, body in _kernels() if "pdl()" in body]
    assert len(early) >= 30  # the scan sees the library's kernels
    for name, head in early:
        promised = set(re.findall(r"__restrict__\s*(\w+)", head))
        assert promised <= TABLES, (name, promised - TABLES)


def test_every_kernel_waits_before_its_first_statement_on_data():
    """What stands before pdl() in a kernel names no data parameter."""
    for name, head, body in _kernels():
        if "pdl()" not in body:
            continue
        before = body[: body.index("pdl()")]
        data = set(re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)\s*[,)]", head)) - TABLES
        used = {d for d in data if re.search(rf"\b{d}\b", before)}
        assert not used, (name, used)

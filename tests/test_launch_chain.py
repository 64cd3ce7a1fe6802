"""Chained kernels (launch_chain.cuh) start while their predecessor still writes.  A
`__restrict__` parameter promises the compiler that nothing else writes the buffer while the
kernel lives, so only tables written before the chain may carry it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "baandi_b200", "csrc")
# operator and projector tables, twiddles, sphere indices, the mixer's fixed metric tables
TABLES = {"tabs", "nls", "twg", "idx", "smooth", "screening"}


def chained_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = open(path).read()
        for m in re.finditer(r"__global__(.*?)\)\s*\{(.*?)\n\}\n", text, re.S):
            if "chain_wait();" in m.group(2):
                name = re.findall(r"(k_\w+)\(", m.group(1))[-1]
                yield os.path.basename(path), name, m.group(1), m.group(2)


def test_chained_kernels_wait_first():
    found = list(chained_kernels())
    assert len(found) > 30
    for path, name, _, body in found:
        assert body.lstrip().startswith("chain_wait();"), (path, name)


def test_restrict_only_on_tables():
    for path, name, signature, body in chained_kernels():
        promised = set(re.findall(r"__restrict__\s+(\w+)", signature))
        assert promised <= TABLES, (path, name, promised - TABLES)
        for target in re.findall(r"__restrict__\s+(\w+)\s*=", body):
            assert target in {"atom_off", "d_off", "d"}, (path, name, target)


def test_every_chained_launch_names_a_chained_kernel():
    names = {name for _, name, _, _ in chained_kernels()}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        for kernel in re.findall(r"launch_chained\(\s*(k_\w+)", open(path).read()):
            assert kernel in names, (os.path.basename(path), kernel)


def test_no_kernel_releases_its_successor_early():
    # blocks of a successor released early run unevenly spread and with the predecessor's L1
    # share: solves of capacities 60 to 128 lost up to a fifth of their speed (launch_chain.cuh)
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        assert "griddepcontrol.launch_dependents" not in open(path).read(), os.path.basename(path)

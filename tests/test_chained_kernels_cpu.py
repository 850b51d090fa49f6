"""The rules of a chained launch (launch_chained in fpg_internal.h), read off
the sources: a kernel that waits for its predecessor inside (chain_begin) does
so before any access to memory, and reads nothing that an earlier kernel of
the stream may have written by a load the compiler may move above that wait --
a parameter marked __restrict__, or a read-only load at an address that does
not itself come from memory."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flexpart-gpu_b200", "csrc")
SOURCES = {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read())
           for p in glob.glob(os.path.join(CSRC, "*.cu*"))}

# The read-only loads of the library: their address is a particle's cell or
# node, which the kernel has loaded before.
FROM_MEMORY = [
    r"__ldg\(q( \+ [12])?\)",                          # ld_cell_hanna: the slot's met cell
    r"__ldg\(a\.wet_cells \+ ",                        # the slot's met cell
    r"__ldg\(pbl \+ pbl_cell_index\(v, p, ",           # the slot's met cell
    r"ld\.global\.nc\.v8\.f32 ",                       # ld_node: a corner of the particle's cell
]


def _kernels():
    """(file, name, parameters, body) of every __global__ function definition."""
    for name, text in SOURCES.items():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)\(([^{;]*?)\)\s*\{",
                             text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield name, m.group(1), m.group(2), text[m.end():end]


def _chained():
    return [k for k in _kernels() if "chain_begin()" in k[3]]


def test_chained_kernels_wait_first_and_take_plain_pointers():
    chained = _chained()
    assert len(chained) >= 25
    for file, name, params, body in chained:
        assert body.strip().startswith("chain_begin();"), (file, name)
        assert "__restrict__" not in params, (file, name)


def test_every_kernel_launched_by_name_in_a_chain_waits():
    chained = {name for _, name, _, _ in _chained()}
    known = {name for _, name, _, _ in _kernels()}
    launched = {n for text in SOURCES.values() for n in re.findall(r"launch_chained\((\w+)", text)} & known
    assert launched and launched <= chained


def test_read_only_loads_take_their_address_from_memory():
    for file, text in SOURCES.items():
        for m in re.finditer(r"__ldg\(|ld\.global\.nc", text):
            assert any(re.match(p, text[m.start():]) for p in FROM_MEMORY), (file, text[m.start():m.start() + 60])

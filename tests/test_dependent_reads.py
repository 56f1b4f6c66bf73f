"""Reads of what an earlier launch wrote, by kernels that start before their predecessor has ended (csrc, `pdl_wait`). Such a kernel may start
while the launch before its predecessor still pulls a buffer's last contents into L1; the read-only path (ld.global.nc: `__ldg`,
skd::ld_ro / ld_stream, and plain reads of `const __restrict__` arguments) may then serve those. So the read-only path is for weights
and tables, and everything else goes through skd::ld_dep or a pointer without `__restrict__`.

Read from the sources: whether a stale line is hit depends on which SM a block lands on."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "skainet_b200", "csrc")

# Never written while kernels that read them are in flight: weights, norms, rotation tables; TurboQuant planes and the
# decode attention's binary16 rows, each appended once, on lines of its own, by a launch that no later one overtakes.
CONSTANT = {"qs", "hdr", "hrow", "codes", "scales", "ql", "qh", "sc", "dd", "w", "wr", "qp", "gamma", "in.gamma", "gains", "cos_t", "sin_t", "cr", "sr", "table",
            "pl.scales", "pl.signs", "kc", "vc", "kb", "vb"}


def kernels(text):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__", text):
        at = text.index("{", m.end())
        head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text[m.end():at])
        depth, end = 0, at
        for end in range(at, len(text)):
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            if depth == 0:
                break
        name = re.search(r"(\w+)\s*\(", head)
        yield name.group(1), head[name.end():], text[at:end]


def first_pointer(text, at):
    """The first name in the argument of a call whose '(' is at `at`, casts and types left out."""
    arg = text[at + 1:at + 200]
    arg = re.sub(r"reinterpret_cast<[^>]*>|\(const [\w ]+\*\)|\(", " ", arg)
    return re.match(r"\s*([\w.]+)", arg).group(1)


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        if os.path.basename(path) == "probe.cu":                # reads what nothing writes
            continue
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", open(path).read())


def test_arguments_of_early_kernels():
    found = []
    for path, text in sources():
        for name, params, body in kernels(text):
            if "pdl_wait" not in body:
                continue
            found += [(path, name, p) for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params) if p not in CONSTANT]
    assert not found


def test_read_only_loads():
    found = []
    for path, text in sources():
        plain = "".join(body for _, _, body in kernels(text) if "pdl_wait" not in body)        # these start when all before them has ended
        for m in re.finditer(r"(?:__ldg|\bld_ro|\bld_stream|\bld_nc_v4)\s*(\()", text):
            if text[max(0, m.start() - 40):m.start()].rstrip().endswith(("uint4", "return")):           # their definitions
                continue
            p = first_pointer(text, m.start(1))
            if p not in CONSTANT and text[m.start() - 20:m.end() + 60] not in plain:
                found.append((path, p))
    assert not found

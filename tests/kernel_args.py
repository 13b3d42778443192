"""Template arguments of the kernels that a timed call has launched, by the names that the sources give the parameters (a mangled name has their values in order)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "marian-dev_b200", "csrc")


def parameters(kernel: str) -> list:
    """The names of a kernel's template parameters, from its source."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                m = re.search(r"template <([^<>]*)>\s*__global__[^;{]*?\b%s\(" % kernel, f.read())
            if m:
                return [p.split("=")[0].split()[-1] for p in m.group(1).split(",")]
    raise AssertionError("no kernel template " + kernel)


def arguments(kernel: str, mangled: str):
    """{parameter: value} of an instantiation, or None where `mangled` is another kernel."""
    m = re.search(r"\d%sI((?:L[a-z]n?\d+E)+)" % kernel, mangled)
    if m is None:
        return None
    values = [int(v.replace("n", "-")) for v in re.findall(r"L[a-z](n?\d+)E", m.group(1))]
    names = parameters(kernel)
    assert len(values) == len(names), (mangled, names)
    return dict(zip(names, values))

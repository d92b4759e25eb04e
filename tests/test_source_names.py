"""A file's own constants do not hide the enumerators of the shared headers: a status word
written through such a name would hold the constant."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pars_gb300", "csrc")


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


def test_constants_do_not_hide_enumerators():
    enumerators = set()
    for header in glob.glob(os.path.join(CSRC, "*.hpp")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        for body in re.findall(r"\benum\s+(?!class\b)\w*\s*(?::\s*\w+\s*)?\{([^}]*)\}", _code(header)):
            enumerators |= set(re.findall(r"(?:^|,)\s*(\w+)", body))
    assert {"async_wait_limit", "async_ok"} <= enumerators
    hidden = []
    for source in glob.glob(os.path.join(CSRC, "*.cu")):
        for name in re.findall(r"\bconstexpr\s+[\w:\s]+?\b(\w+)\s*=", _code(source)):
            if name in enumerators:
                hidden.append((os.path.basename(source), name))
    assert not hidden, hidden

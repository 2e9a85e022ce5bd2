"""Rules of the device code that a wrong kernel would break only when something
else has already failed, checked on the source (no GPU needed)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "speccodelib_gb300", "csrc")


def kernels():
    """(name, body) of every __global__ function in the headers."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\s*\([^;{]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            out.append((m.group(1), text[m.end():i]))
    return out


def test_grouped_kernels_exit_uniformly():
    """A thread group's named barrier counts its threads whether or not some have
    left, so a kernel that uses one does not return on a thread's own view of the
    error word or of a timed-out wait: the CTA agrees first."""
    grouped = [(n, b) for n, b in kernels() if re.search(r"ZG::Engine|AdjGrpCfg|ZiCfg", b)]
    names = {n for n, _ in grouped}
    assert {"zinv_phi_tma_kernel", "zfwd_tma_kernel", "zfwd_zinv_tma_kernel", "zfwd_adj_group_kernel"} <= names
    for name, body in grouped:
        own = re.findall(r"if \((?:!mbar_wait_bounded|launch_failed)\([^;]*return;", body)
        assert not own, (name, own)

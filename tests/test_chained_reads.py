"""The step's kernels may be resident while the kernels before them in the chain still write, so what any of
them writes may not be read through the read-only path (__ldg), whose data must not change while the
kernel lives. Checked on the source: no run can show that the order always holds."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lydion_b200", "csrc",
                   "lyd_kernels.cu")
# what k_advect, k_freq and k_reduce write, by the names of their argument blocks
WRITTEN = ("J", "Hr", "HZ", "Jo", "Hro", "HZo", "Jin", "Hrin", "HZin", "Jold", "Jout", "Hrout", "HZout", "dru_r",
           "dru_Z", "f_r", "f_Z", "Fkp", "Fk", "Fkm", "tape", "partials", "kwin", "kwin_copy", "colsum", "cnt", "diag",
           "last", "step_counter", "done")


def _calls(text, name):
    """The argument texts of every call of `name`."""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_nothing_a_step_kernel_writes_is_read_through_ldg():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    # `ld` is the frequency kernel's per-cell loader, an __ldg inside
    assert "auto ld = [&](const double *p, bool need) { return (v && need && p) ? __ldg(p + cc) : 0.0; };" in text
    bad = [c for f in ("__ldg", "ld") for c in _calls(text, f)
           if re.search(r"\ba\.(%s)\b" % "|".join(WRITTEN), c)]
    assert not bad, bad

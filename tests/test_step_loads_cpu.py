"""Step kernels are launched with overlap: a kernel's lifetime begins while
the kernels ahead of it still write.  Read-only loads (__ldg, ld.global.nc)
are defined only for data nobody writes during that lifetime, so they may
name the potential tables, which are uploaded before any step, and nothing
that a refresh, a list build or a density pass writes."""
import glob
import os
import re

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fmd_gb300", "csrc", "cuda")
# uploaded by fmdg_set_eam (`row`, `tpr`: pointers into them)
TABLES = {"g.pkd_phi", "g.pkd_rho", "g.pkd_pr", "g.pkf_pr", "tpr", "row"}


def _loads():
    for path in sorted(glob.glob(os.path.join(CUDA, "*.cu*"))):
        code = re.sub(r"//[^\n]*", "", open(path).read())
        code = re.sub(r"reinterpret_cast<[^>]*>\(", "", code)
        for m in re.finditer(r"\b(?:__ldg|ld_row32)\(\s*([\w.]+)", code):
            if m.group(1) != "const":       # (the definition of ld_row32)
                yield os.path.basename(path), m.group(1)


def test_read_only_loads_name_tables_only():
    loads = list(_loads())
    assert loads
    assert [l for l in loads if l[1] not in TABLES] == []


def test_one_read_only_asm_load():
    n = sum(open(p).read().count('"ld.global.nc') for p in glob.glob(os.path.join(CUDA, "*.cu*")))
    assert n == 1       # ld_row32
    for name in ("g.pkd_pr", "g.pkf_pr"):
        # what `row` and `tpr` point into
        assert any(re.search(r"(eam_pair_row\(|tpr = )%s\b" % re.escape(name), open(p).read())
                   for p in glob.glob(os.path.join(CUDA, "*.cu*")))

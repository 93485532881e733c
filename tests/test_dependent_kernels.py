"""Kernels that start while the one before them ends (dependent_begin): what an
earlier kernel may still be writing is not read through the read-only path,
whose data has to be unchanged for the kernel's whole life.  So a const
__restrict__ parameter or an operand of __ldg is a table made at set-up, the
matrix, its factors or the user's data; a parameter without a const that a
kernel only reads counts too (the basis and the vector of the dots)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "goma_gb300",
                    "csrc")
# tables; the matrix and the factors; the basis (other kernels lie between the
# one that writes a vector and its first use); the network's training data
UNCHANGED = {
    "*": {"tb", "gtb", "elems", "rowptr", "colidx", "groups", "tseg", "tbeg", "tend", "tptr",
          "active"},
    "assemble_sf_kernel": {"d"},  # of tb
    "spmv_kernel": {"vals"},
    "line_sweep_kernel": {"vals", "b"},  # b: read by ld_relaxed
    "gs_kernel": {"V"},
    "loss_grad_kernel": {"T", "mask"},
    "gather_rows_kernel": {"idx", "X", "T", "K"},
}
ONLY_READ = {"gs_kernel": {"w"}, "seg_gs_kernel": {"w"}}  # in the dots


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^\n]*\)\s+)?(\w+)\(", text):
            end = text.index("\n}\n", m.end())
            body = text.index("{", text.index(")", m.end()))
            if "dependent_begin()" in text[body:end]:
                yield m.group(1), text[m.end():body], text[body:end]


def test_operands_of_earlier_kernels_are_not_read_only():
    found = dict((name, (params, body)) for name, params, body in kernels())
    assert {"spmv_kernel", "gs_kernel", "seg_scale_kernel", "mlp_gemm_kernel", "adam_kernel",
            "assemble_2d_kernel", "line_sweep_kernel"} <= set(found)
    bad = []
    for name, (params, body) in found.items():
        ok = UNCHANGED["*"] | UNCHANGED.get(name, set())
        bad += [(name, p) for p in re.findall(r"const \w+ \*__restrict__ (\w+)", params)
                if p not in ok]
        bad += [(name, p) for p in re.findall(r"\w+ \*__restrict__ (\w+)", params)
                if p in ONLY_READ.get(name, set())]
        bad += [(name, p) for p in re.findall(r"__ldg\(&?(\w+)", body) if p not in ok]
    spmv = open(os.path.join(CSRC, "gb_solve.cu")).read()
    spmv = spmv[spmv.index("void spmv_group("):spmv.index("spmv_kernel(")]
    bad += [("spmv_group", p) for p in re.findall(r"__ldg\((\w+)|__restrict__ (x)\b", spmv)]
    assert not bad, bad

"""Kernel attributes (shared memory allowed) belong to a device, the runtime is kept per device: what a
kernel's set-up remembers must be, too.  One GPU cannot show the difference, so the source is read: no
function keeps a flag or an occupancy for the whole process, and the holder keeps one per device."""
import glob
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rqcopt_hpc_b200", "csrc")


def test_no_set_up_is_remembered_for_the_whole_process():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for n, line in enumerate(open(path), 1):
            if re.match(r"\s+static (bool|int) \w+ = (false|0);", line):
                found.append(f"{os.path.basename(path)}:{n}")
    assert not found


def test_the_holder_keeps_a_value_per_device(tmp_path):
    header = open(os.path.join(CSRC, "rqc_runtime.h")).read()
    body = re.search(r"struct PerDevice\n\{.*?\n\};", header, re.S).group(0)
    (tmp_path / "t.cpp").write_text("struct Runtime { int device; };\n" + body + """
int main()
{
	static PerDevice p;
	Runtime a{0}, b{1}, c{7};
	p[a] = 3;
	if (p[b] != 0 || p[c] != 0) return 1;
	p[c] = 5;
	return p[a] == 3 && p[b] == 0 && p[c] == 5 ? 0 : 2;
}
""")
    subprocess.run(["g++", "-std=c++17", "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0

"""The slots of the batched SVD's plan memory (vecjac_gb300/csrc/plan_slots.h): a launch captured into a
graph keeps its slot until the graph is gone, however many launches come later, and a slot of
launches that run at once is handed out again only after its holder is done with it."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_slots(tmp_path):
    exe = str(tmp_path / "plan_slots_host")
    r = subprocess.run(["g++", "-O1", "-std=c++17", os.path.join(HERE, "plan_slots_host.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.stdout == "ok\n", r.stdout

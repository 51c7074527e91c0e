"""Cluster sizes of the resident classes of one batch (cluster_share.hpp): the
classes run beside each other, so together they must not ask for more SMs than
there are while smaller clusters would fit."""

import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "qoraphasecu_b200" / "csrc"

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "cluster_share.hpp"
// argv: SMs, clusters of 16 at once, then side and starts of every class
int main(int argc, char** argv) {
  const int sms = std::atoi(argv[1]), large = std::atoi(argv[2]);
  std::vector<qpb::ClusterClaim> claims;
  for (int i = 3; i + 1 < argc; i += 2) {
    qpb::ClusterClaim c{std::atoi(argv[i]), std::atoi(argv[i + 1]), {}};
    for (auto s : qpb::cluster_sizes(c.side)) c.room.push_back(s.ctas == 16 ? large : sms / s.ctas);
    claims.push_back(c);
  }
  for (int s : qpb::share_clusters(claims, sms)) std::printf("%d ", s);
}
"""


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    out = tmp_path_factory.mktemp("share")
    (out / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++20", "-I", str(CSRC), str(out / "main.cpp"), "-o",
                    str(out / "share")], check=True)

    def run(*classes, sms=148, large=8):
        args = [str(a) for c in classes for a in c]
        done = subprocess.run([str(out / "share"), str(sms), str(large), *args], check=True,
                              capture_output=True, text=True)
        return [int(s) for s in done.stdout.split()]

    return run


@pytest.mark.parametrize("classes", [
    [(64, 4), (128, 4), (256, 4)], [(64, 18), (128, 8)], [(64, 8), (256, 8)], [(64, 8), (128, 8)],
    [(64, 2), (128, 2), (256, 2)], [(64, 100), (128, 9)], [(128, 30), (256, 8)],
])
def test_classes_fit_beside_each_other(share, classes):
    sizes = share(*classes)
    assert sum(starts * ctas for (_, starts), ctas in zip(classes, sizes)) <= 148
    assert sum(starts for (_, starts), ctas in zip(classes, sizes) if ctas == 16) <= 8


def test_the_slowest_class_keeps_its_clusters(share):
    assert share((64, 4), (128, 4), (256, 4))[2] == 16
    assert share((64, 18), (128, 8)) == [1, 16]


def test_idle_sms_are_used(share):
    assert share((64, 2), (128, 2)) == [8, 16]


def test_more_starts_than_any_size_fits(share):
    sizes = share((64, 400), (128, 300), (256, 90))
    assert sizes[0] in (1, 2, 4, 8) and sizes[1] in (2, 4, 8, 16) and sizes[2] in (8, 16)

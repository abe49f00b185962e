"""The host view dumps the reverse passes that run: parameters are shared by the samples and staged in
every reverse sweep, so the sources of a batch are those of one sample (CPU)."""
from mossquantum_b200 import workloads as W
from tests.test_schedule import schedule_info


def test_batch_sources_stage_parameters(monkeypatch, tmp_path):
    monkeypatch.setenv("MB_JIT_DUMP_ADJOINT", "1")
    got = {}
    for B in (1, 4):
        d = tmp_path / str(B)
        d.mkdir()
        monkeypatch.setenv("MB_JIT_DUMP", str(d))
        schedule_info(W.hea_circuit(14, 2), 14, t=10, nsamples=B)
        got[B] = [p.read_text() for p in sorted(d.glob("adj_*.cu"))]
    assert len(got[1]) and len(got[1]) == len(got[4])
    for one, many in zip(got[1], got[4]):
        assert ("smat" in one) == ("smat" in many) and one.count("tab[") == many.count("tab[")

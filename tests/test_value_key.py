"""Circuits remember a checked compilation by value: any change of what they hold is seen, however it
was made (CPU)."""
import numpy as np
import pytest

import mossquantum_b200 as mq


def circuit():
    c = mq.QCircuit([mq.RxGate(1, 0.3, isparas=True), mq.RzGate(2, 0.4), mq.CNOTGate(1, 2),
                     mq.QuantumGate(3, np.eye(2)), mq.Depolarizing(2, 0.1)])
    return mq.QCircuit([c, mq.RyGate(3, 0.1, isparas=True)])


def change_flag(c):
    c[0][0].isparas[0] = False


def change_kraus(c):
    c[0][4].kraus[0][0, 0] *= 0.5


def change_matrix(c):
    c[0][3].data[1, 1] = -1


def change_position(c):
    c[0][2].pos = (2, 1)


def change_frozen(c):
    c[0][1].paras[0] = 0.5


def change_type(c):
    c[0].items[2] = mq.CZGate(1, 2)


def change_position_to_list(c):
    c[0][2].pos = [1, 2]


CHANGES = [change_flag, change_kraus, change_matrix, change_position, change_frozen, change_type, change_position_to_list,
           lambda c: c[0].push(mq.XGate(1)), lambda c: c.items.pop()]


@pytest.mark.parametrize("change", CHANGES)
def test_changes_are_seen(change):
    c, marker = circuit(), object()
    assert c.known(3, c.value_key()) is None
    c.remember(3, marker, c.value_key())
    assert c.known(3, c.value_key()) == (marker, True) and c.known(4, c.value_key()) is None
    c.reset_parameters([1.0, 2.0])                  # active values are not part of it
    assert c.known(3, c.value_key()) == (marker, True)
    change(c)
    assert c.known(3, c.value_key()) is None


def test_unknown_types_are_not_remembered():
    for gate in (mq.RxGate(1, 0.2, isparas=True).adjoint(), mq.FSIMGate(1, 2, [0.1] * 5), mq.CONTROLGate(1, 2, np.eye(2))):
        c = mq.QCircuit([gate])
        c.remember(2, object(), c.value_key())
        assert c.known(2, c.value_key()) is None


def test_operator_checks_follow_the_terms():
    op = mq.QubitsOperator([mq.QubitsTerm([1, 3], ["X", "Z"], 0.5), mq.QubitsTerm([2], ["Y"], -1.0)])
    assert op.nqubits() == 3 and op.is_hermitian()
    op.terms[1].op[0][0, 1] = 3.0
    assert not op.is_hermitian()
    op.terms[1].op[0][0, 1] = -1j
    assert op.is_hermitian()
    op.add(mq.QubitsTerm([1, 2, 4], ["Z"] * 3, 1j))
    assert op.nqubits() == 4 and not op.is_hermitian()
    pair = mq.QubitsOperator([mq.QubitsTerm([1], ["+"], 1.0), mq.QubitsTerm([1], ["-"], 1.0)])
    assert pair.is_hermitian() and mq.QubitsOperator([]).is_hermitian()

: A leak that counts the evaluations of its BREAKPOINT and sums its charge, written for the tests
: of steps that are solved twice: both fields feed the next evaluation.
NEURON {
    POINT_PROCESS UserCounter
    NONSPECIFIC_CURRENT i
    RANGE g, e, n, q, i
}

UNITS {
    (nA) = (nanoamp)
    (mV) = (millivolt)
    (uS) = (microsiemens)
}

PARAMETER {
    g = 0.002 (uS) <0,1e9>
    e = -60 (mV)
}

ASSIGNED {
    v (mV)
    i (nA)
    n
    q (pC)
}

INITIAL {
    n = 0
    q = 0
}

BREAKPOINT {
    i = g*(v - e)
    n = n + 1
    q = q + i*dt
}

// When a captured step's calls launch several steps in one graph, and of how many
// steps that graph is (host code; sg_step).
#pragma once

// Between two graph launches the stream idles for 3.5 to 5 us; inside a graph
// kernels follow each other in 0.1 to 0.3. 30 steps of 2 916 LJ particles take
// 726 us in graphs of one step and 631 in graphs of 15, 20 ECP steps of 65 536
// particles 1229 and 1132, 10 chain steps of 96 000 beads 928 and 911. The graph
// holds a whole fraction of the steps that the caller asks for at a time, at most
// SG_GRAPH_STEPS: past that a gap is less than 0.3 us a step.
// Putting it together costs the host 2.5 to 2.6 us a node (10 steps of four kernels
// 105 us, 16 of them 166, 16 of six 235), what the gaps of some forty steps take. So
// it is made for a call whose own gaps cost as much, or once those of the calls
// since the capture have: a program that changes its configuration or its box every
// few calls does not pay for graphs that it throws away, and none pays more for
// them than for the gaps. LJ, us a configuration, made by its second call (or
// one of 64 steps) / by this rule: two calls of 10 steps 501 / 380, four of 20 1316 /
// 1357, eight 2380 / 2417, twenty of 30 8225 / 8172, one of 64 1092 / 1075. It is
// replaced only by one four times as long, by the same rule.
#define SG_GRAPH_STEPS 16
#define SG_GRAPH_GAP_US 4
#define SG_GRAPH_NODE_US 3

struct GraphSteps {
    int steps = 0;         // steps of the graph of several that there is, 0: none
    long long gaps = 0;    // graph launches since the capture, or since that graph was made

    // launches that nsteps take with what there is
    long long launches(int nsteps) const { return steps > 1 ? nsteps / steps + nsteps % steps : nsteps; }
    // steps of the graph to make before nsteps of kernels nodes each, 0: none
    int wanted(int nsteps, int kernels) const {
        if (nsteps < 2) return 0;
        const int want = nsteps / ((nsteps + SG_GRAPH_STEPS - 1) / SG_GRAPH_STEPS);
        if (want < 2 || want < 4 * steps) return 0;
        const long long now = launches(nsteps), most = gaps > now ? gaps : now;
        return SG_GRAPH_GAP_US * most >= (long long)SG_GRAPH_NODE_US * kernels * want ? want : 0;
    }
    void made(int n) {
        steps = n;
        gaps = 0;
    }
};

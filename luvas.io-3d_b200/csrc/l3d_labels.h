/*
 * Component labels by union-find: the steps of the component kernels (mesh.cu), over any memory of
 * labels, so that the host can run them under every order of their loads and stores.
 *
 * label[v] leads from v to vertices of ever lower rank until a root, a vertex that is its own label.  Mem
 * gives load(v), store(v, l) and swap(v, from, to) (compare-and-swap, true when done), each of them one
 * indivisible access to one word.
 */
#ifndef L3D_LABELS_H
#define L3D_LABELS_H

#include <stdint.h>

#include "l3d_fmath.h"

#ifdef __CUDACC__
#define L3D_LABELS __device__ __forceinline__
#else
#define L3D_LABELS static inline
#endif

constexpr int kLabelGuard = 1 << 24;  /* steps along labels, each to a vertex of lower rank */

/* A vertex's rank among roots: the random numbers' hash (l3d_fmath.h).  It is a bijection (an affine map
 * with an odd factor, a xorshift by an amount that the top bits, which it keeps, give, a product with an
 * odd number, another xorshift), so ranks are distinct; and it mixes, so that linking a mesh's vertices
 * in their scan order does not build long chains (linked by index, 74 thousand faces took 93 us). */
L3D_HD uint32_t l3d_label_rank(uint32_t v) { return l3d_pcg(v); }

/* The root of v while components are joined; every vertex passed is pointed at its successor's successor.
 * Such a store can overwrite a shorter path that another thread stored: the vertex still leads to its
 * root, so this holds only while no thread takes a label for a root without looking (l3d_label_flatten). It
 * never overwrites a root's hook: a root is only written by the compare-and-swap that ends its being
 * one. */
template <class Mem>
L3D_LABELS uint32_t l3d_label_root_halving(Mem& m, uint32_t v, int* err) {
    uint32_t p = m.load(v);
    for (int guard = 0; p != v; guard++) {
        const uint32_t g = m.load(p);
        if (g == p) break;
        if (guard >= kLabelGuard) {
            *err = 1;
            break;
        }
        m.store(v, g);
        v = p;
        p = g;
    }
    return p;
}

/* Joins the components of a and b: the root of higher rank onto the other. */
template <class Mem>
L3D_LABELS void l3d_label_unite(Mem& m, uint32_t a, uint32_t b, int* err) {
    for (int guard = 0; guard < kLabelGuard; guard++) {
        a = l3d_label_root_halving(m, a, err);
        b = l3d_label_root_halving(m, b, err);
        if (a == b) return;
        const bool a_up = l3d_label_rank(a) > l3d_label_rank(b);
        const uint32_t hi = a_up ? a : b, lo = a_up ? b : a;
        if (m.swap(hi, hi, lo)) return;
    }
    *err = 1;
}

/* label[v] = the root of v, once nothing is joined any more.  The walk only loads, and each label has one
 * writer, its own vertex: what others read there meanwhile is the old successor or the root, both on the
 * way to the same root.  (Shortening paths here would let a thread that walks past v put an inner vertex
 * back after v's own thread has stored the root, and v's faces would count as a component apart.) */
template <class Mem>
L3D_LABELS void l3d_label_flatten(Mem& m, uint32_t v, int* err) {
    uint32_t root = v;
    for (int guard = 0;; guard++) {
        const uint32_t p = m.load(root);
        if (p == root) break;
        root = p;
        if (guard >= kLabelGuard) {
            *err = 1;
            break;
        }
    }
    m.store(v, root);
}

#endif

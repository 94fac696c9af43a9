// The device's replay of recorded leaf moves into the broadphase tree:
// the operations of m3_tree.h (dynamic_tree.c:92-358) carried out by one
// warp, with the same nodes as a result, byte for byte.
//
// What bounds it: a world's moves are a serial chain (each move's walks
// read what the move before wrote) run by one warp, whose instructions
// mostly wait for the one before (3.7 cycles each, L1 hits 99 % of the
// loads of a 2048-body world), so the time is moves x levels x the
// instructions of a level, not bandwidth.  What shortens the chain:
//
//  * A refit stops at the first node that it leaves as it found it.
//    Every node above then sees unchanged children, and its own refit
//    would change nothing unless it is out of balance (an insertion that
//    stops at an inner node can leave one such node behind).  The nodes
//    out of balance are few; the warp keeps their list, one per lane, and
//    a walk goes on when one of their boxes encloses the node it would
//    stop at.  Of 10 to 14 levels a refit visits 3 to 5.
//  * A refit's level is one load deep: lane k < 6 owns bound k of every
//    record, links and heights are read by all lanes, the parent's record
//    is asked for beside the sibling's.
//  * The descent looks one level ahead: four lanes hold the two children
//    of both children, so a level's decision only picks records already
//    on their way.
//
// A leaf and its parent node keep their ids through a move: a removal
// frees the parent, then the leaf, and the insertion takes the leaf, then
// the parent, from the same free list, whose head ends where it began.
#ifndef M3_TREEWALK_CUH
#define M3_TREEWALK_CUH

#include "m3_tree.h"

#define M3_FULL_WARP 0xFFFFFFFFu

// What the scratch remembers of a world's tree between launches: the mode
// (word 0) and the nodes out of balance (words 1 to 32, -1: none).  Walks
// stop early only in the TRACKED mode; FULL walks go to the root, as they
// must when a box holds a NaN or a negative zero (min and max then depend
// on the operands' order), when a restored tree's inner boxes are not the
// union of their children's, or when the list would overflow.
#define M3_TREE_STATE_WORDS 33
#define M3_TREE_TRACKED 1
#define M3_TREE_FULL 2

// A box whose unions do not depend on the operands' order.
__device__ __forceinline__ bool m3TreePlainBox(const double* lo, const double* hi)
{
    bool plain = true;
    for (int32_t k = 0; k < 3; ++k)
    {
        plain = plain && lo[k] == lo[k] && hi[k] == hi[k] &&
                !(lo[k] == 0.0 && __double_as_longlong(lo[k]) < 0) &&
                !(hi[k] == 0.0 && __double_as_longlong(hi[k]) < 0);
    }
    return plain;
}

// A 72-byte record as its links: {parent, child1}, {child2, userData},
// {height, pad} after the six bounds.
struct m3TreeLinks
{
    int32_t parent;
    int32_t child1;
    int32_t child2;
    int32_t height;
};

struct m3TreeWarp
{
    m3TreeNode* nodes;
    int32_t capacity;
    int32_t root;  // the same in every lane
    int32_t lane;
    int32_t bound; // the bound of a record this lane owns
    int32_t unbalanced; // one node out of balance, or M3_TREE_NULL
    bool tracked;  // walks may stop early

    __device__ __forceinline__ double Bound(int32_t i) const
    {
        return ((const double*)(nodes + i))[bound];
    }
    __device__ __forceinline__ m3TreeLinks Links(int32_t i) const
    {
        const int2* q = (const int2*)((const double*)(nodes + i) + 6);
        const int2 a = q[0];
        const int2 b = q[1];
        m3TreeLinks l;
        l.parent = a.x;
        l.child1 = a.y;
        l.child2 = b.x;
        l.height = nodes[i].height;
        return l;
    }
    // `first` before `second`, as m3TreeUnion orders them.
    __device__ __forceinline__ double Union(double first, double second) const
    {
        const bool takeFirst = bound < 3 ? first < second : first > second;
        return takeFirst ? first : second;
    }
    // The lanes that own a bound write it; links are written by every lane
    // (the same value), so each lane later reads its own write.
    __device__ __forceinline__ void PutBound(int32_t i, double x) const
    {
        if (lane < 6)
        {
            ((double*)(nodes + i))[lane] = x;
        }
    }

    __device__ __forceinline__ void Balanced(int32_t i)
    {
        unbalanced = unbalanced == i ? M3_TREE_NULL : unbalanced;
    }
    __device__ __forceinline__ void Unbalanced(int32_t i)
    {
        const uint32_t room = __ballot_sync(M3_FULL_WARP, unbalanced == M3_TREE_NULL);
        if (room == 0)
        {
            tracked = false;
        }
        else if (lane == __ffs((int)room) - 1)
        {
            unbalanced = i;
        }
    }

    // Whether a node out of balance may stand above node i (its box
    // encloses i's, as every ancestor's does).
    __device__ __forceinline__ bool UnbalancedAbove(int32_t i) const
    {
        if (__ballot_sync(M3_FULL_WARP, unbalanced != M3_TREE_NULL) == 0)
        {
            return false;
        }
        __syncwarp();
        bool above = false;
        if (unbalanced != M3_TREE_NULL)
        {
            const m3TreeNode& u = nodes[unbalanced];
            const m3TreeNode& n = nodes[i];
            above = u.lo[0] <= n.lo[0] && u.lo[1] <= n.lo[1] && u.lo[2] <= n.lo[2] &&
                    n.hi[0] <= u.hi[0] && n.hi[1] <= u.hi[1] && n.hi[2] <= u.hi[2];
        }
        return __any_sync(M3_FULL_WARP, above);
    }

    // m3TreeRefit from node `index` (links n, own bound `box`), whose
    // child `from` has bound `fromBox` and height `fromHeight`; `changed`
    // says that the node's record is new whatever its refit gives.
    __device__ void Refit(int32_t index, m3TreeLinks n, double box, int32_t from, double fromBox,
                          int32_t fromHeight, bool changed)
    {
        bool toRoot = !tracked;
        for (int32_t guard = 0; guard < capacity; ++guard)
        {
            const bool fromFirst = n.child1 == from;
            const int32_t other = fromFirst ? n.child2 : n.child1;
            const double otherBox = Bound(other);
            const int32_t otherHeight = nodes[other].height;
            const int32_t up = n.parent;
            m3TreeLinks upLinks = n;
            double upBox = 0.0;
            if (up != M3_TREE_NULL)
            {
                upLinks = Links(up);
                upBox = Bound(up);
            }
            const double c1 = fromFirst ? fromBox : otherBox;
            const double c2 = fromFirst ? otherBox : fromBox;
            const int32_t h1 = fromFirst ? fromHeight : otherHeight;
            const int32_t h2 = fromFirst ? otherHeight : fromHeight;
            const int32_t balance = h2 - h1;
            if (n.height >= 2 && (balance > 1 || balance < -1))
            {
                // m3TreeRotate: the taller child p rises, `index` becomes
                // its first child.
                const bool right = balance > 1;
                const int32_t p = right ? n.child2 : n.child1;
                const double q = right ? c1 : c2;
                const int32_t qHeight = right ? h1 : h2;
                const m3TreeLinks P = Links(p);
                const double p1 = Bound(P.child1);
                const double p2 = Bound(P.child2);
                const int32_t p1Height = nodes[P.child1].height;
                const int32_t p2Height = nodes[P.child2].height;
                const bool firstTaller = p1Height > p2Height;
                const int32_t keep = firstTaller ? P.child1 : P.child2;
                const int32_t move = firstTaller ? P.child2 : P.child1;
                const double keepBox = firstTaller ? p1 : p2;
                const double moveBox = firstTaller ? p2 : p1;
                const int32_t keepHeight = firstTaller ? p1Height : p2Height;
                const int32_t moveHeight = firstTaller ? p2Height : p1Height;
                const double aBox = Union(q, moveBox);
                const double pBox = Union(aBox, keepBox);
                const int32_t aHeight = 1 + m3TreeMaxI(qHeight, moveHeight);
                const int32_t pHeight = 1 + m3TreeMaxI(aHeight, keepHeight);
                nodes[p].parent = up;
                nodes[p].child1 = index;
                nodes[p].child2 = keep;
                nodes[p].height = pHeight;
                PutBound(p, pBox);
                nodes[index].parent = p;
                if (right)
                {
                    nodes[index].child2 = move;
                }
                else
                {
                    nodes[index].child1 = move;
                }
                nodes[index].height = aHeight;
                PutBound(index, aBox);
                nodes[move].parent = index;
                if (up == M3_TREE_NULL)
                {
                    root = p;
                }
                else if (upLinks.child1 == index)
                {
                    nodes[up].child1 = p;
                    upLinks.child1 = p;
                }
                else
                {
                    nodes[up].child2 = p;
                    upLinks.child2 = p;
                }
                Balanced(index);
                Balanced(p);
                const int32_t aTilt = qHeight - moveHeight;
                const int32_t pTilt = aHeight - keepHeight;
                if (aTilt > 1 || aTilt < -1)
                {
                    Unbalanced(index);
                }
                if (pTilt > 1 || pTilt < -1)
                {
                    Unbalanced(p);
                }
                if (up == M3_TREE_NULL)
                {
                    return;
                }
                toRoot = toRoot || !tracked;
                from = p;
                fromBox = pBox;
                fromHeight = pHeight;
                index = up;
                n = upLinks;
                box = upBox;
                changed = false;
                continue;
            }
            const int32_t height = 1 + m3TreeMaxI(h1, h2);
            const double fit = Union(c1, c2);
            const bool differs =
                lane < 6 && __double_as_longlong(fit) != __double_as_longlong(box);
            changed = __any_sync(M3_FULL_WARP, differs) || height != n.height || changed;
            if (changed)
            {
                PutBound(index, fit);
                nodes[index].height = height;
            }
            if (up == M3_TREE_NULL)
            {
                return;
            }
            if (!changed && !toRoot)
            {
                if (!UnbalancedAbove(index))
                {
                    return;
                }
                toRoot = true;
            }
            from = index;
            fromBox = fit;
            fromHeight = height;
            index = up;
            n = upLinks;
            box = upBox;
            changed = false;
        }
    }

    // What the descent knows of a candidate node: the area of its union
    // with the new box, its own area, its links.
    struct Candidate
    {
        int32_t id;
        int32_t child1;
        int32_t child2;
        int32_t height;
        double unionArea;
        double area;
    };
    __device__ __forceinline__ Candidate Look(int32_t i, const double* lo, const double* hi) const
    {
        const m3TreeNode& n = nodes[i];
        Candidate c;
        c.id = i;
        const int2* q = (const int2*)((const double*)&n + 6);
        c.child1 = q[0].y;
        c.child2 = q[1].x;
        c.height = n.height;
        double ulo[3];
        double uhi[3];
        m3TreeUnion(n.lo, n.hi, lo, hi, ulo, uhi);
        c.unionArea = m3TreeArea(ulo, uhi);
        c.area = m3TreeArea(n.lo, n.hi);
        return c;
    }

    // m3TreeInsert's descent for the box [lo, hi]: the sibling the new
    // leaf pairs with, its height, its parent and whether it is the
    // parent's first child.  False only for a malformed tree.
    __device__ bool Descend(const double* lo, const double* hi, int32_t* sibling,
                            int32_t* siblingHeight, int32_t* parent, bool* firstChild) const
    {
        const int32_t role = lane & 3;
        const int32_t side = role >> 1;
        const Candidate top = Look(root, lo, hi);
        int32_t index = root;
        int32_t height = top.height;
        double unionArea = top.unionArea;
        double area = top.area;
        *parent = M3_TREE_NULL;
        *firstChild = true;
        int32_t pick = 0;
        Candidate mine = top;
        if (height > 0)
        {
            mine = Look((role & 1) != 0 ? top.child2 : top.child1, lo, hi);
        }
        for (int32_t guard = 0; height > 0; ++guard)
        {
            if (guard >= capacity)
            {
                return false;
            }
            // The two children, held by lanes 2 pick and 2 pick + 1, and
            // this lane's grandchild of them.
            const int32_t src = 2 * pick;
            const int32_t c1 = __shfl_sync(M3_FULL_WARP, mine.id, src);
            const int32_t c2 = __shfl_sync(M3_FULL_WARP, mine.id, src + 1);
            const int32_t h1 = __shfl_sync(M3_FULL_WARP, mine.height, src);
            const int32_t h2 = __shfl_sync(M3_FULL_WARP, mine.height, src + 1);
            const int32_t g1 = __shfl_sync(M3_FULL_WARP, mine.child1, src + side);
            const int32_t g2 = __shfl_sync(M3_FULL_WARP, mine.child2, src + side);
            const double union1 = __shfl_sync(M3_FULL_WARP, mine.unionArea, src);
            const double union2 = __shfl_sync(M3_FULL_WARP, mine.unionArea, src + 1);
            const double area1 = __shfl_sync(M3_FULL_WARP, mine.area, src);
            const double area2 = __shfl_sync(M3_FULL_WARP, mine.area, src + 1);
            // A leaf child has no children: its lanes look at the leaf.
            const int32_t leafOr = side != 0 ? c2 : c1;
            const int32_t sideHeight = side != 0 ? h2 : h1;
            const int32_t grand = sideHeight == 0 ? leafOr : (role & 1) != 0 ? g2 : g1;
            mine = Look(grand, lo, hi);
            const double here = 2.0 * unionArea;
            const double inherited = 2.0 * (unionArea - area);
            const double cost1 = h1 == 0 ? union1 + inherited : union1 - area1 + inherited;
            const double cost2 = h2 == 0 ? union2 + inherited : union2 - area2 + inherited;
            if (here < cost1 && here < cost2)
            {
                break;
            }
            pick = cost1 < cost2 ? 0 : 1;
            *parent = index;
            *firstChild = pick == 0;
            index = pick == 0 ? c1 : c2;
            height = pick == 0 ? h1 : h2;
            unionArea = pick == 0 ? union1 : union2;
            area = pick == 0 ? area1 : area2;
        }
        *sibling = index;
        *siblingHeight = height;
        return true;
    }

    // One move: the leaf `leaf` of `shape` leaves the tree and comes back
    // with the box at `fat` (six bounds).  False for a malformed tree.
    __device__ bool Move(int32_t leaf, int32_t shape, const double* fat)
    {
        const double mine = fat[bound];
        double lo[3];
        double hi[3];
        for (int32_t k = 0; k < 3; ++k)
        {
            lo[k] = fat[k];
            hi[k] = fat[k + 3];
        }
        int32_t parent = M3_TREE_NULL;
        if (leaf != root)
        {
            parent = nodes[leaf].parent;
            const m3TreeLinks P = Links(parent);
            const int32_t sibling = P.child1 == leaf ? P.child2 : P.child1;
            const int32_t grand = P.parent;
            Balanced(parent);
            nodes[sibling].parent = grand;
            if (grand == M3_TREE_NULL)
            {
                root = sibling;
            }
            else
            {
                m3TreeLinks G = Links(grand);
                const double box = Bound(grand);
                if (G.child1 == parent)
                {
                    G.child1 = sibling;
                    nodes[grand].child1 = sibling;
                }
                else
                {
                    G.child2 = sibling;
                    nodes[grand].child2 = sibling;
                }
                Refit(grand, G, box, sibling, Bound(sibling), nodes[sibling].height, false);
            }
            // The descent's lanes read bounds other lanes wrote.
            __syncwarp();
            int32_t under = M3_TREE_NULL;
            int32_t pairHeight = 0;
            int32_t pair = M3_TREE_NULL;
            bool firstChild = true;
            if (!Descend(lo, hi, &pair, &pairHeight, &under, &firstChild))
            {
                return false;
            }
            // The parent node takes the sibling's place.
            m3TreeNode& N = nodes[parent];
            N.parent = under;
            N.child1 = pair;
            N.child2 = leaf;
            N.userData = -1;
            N.height = pairHeight + 1;
            N.pad = 0;
            nodes[pair].parent = parent;
            if (under == M3_TREE_NULL)
            {
                root = parent;
            }
            else if (firstChild)
            {
                nodes[under].child1 = parent;
            }
            else
            {
                nodes[under].child2 = parent;
            }
            m3TreeLinks links;
            links.parent = under;
            links.child1 = pair;
            links.child2 = leaf;
            links.height = pairHeight + 1;
            PutLeaf(leaf, parent, shape, mine);
            Refit(parent, links, 0.0, leaf, mine, 0, true);
            return true;
        }
        PutLeaf(leaf, parent, shape, mine);
        return true;
    }

    __device__ __forceinline__ void PutLeaf(int32_t leaf, int32_t parent, int32_t shape,
                                            double mine) const
    {
        m3TreeNode& L = nodes[leaf];
        L.parent = parent;
        L.child1 = M3_TREE_NULL;
        L.child2 = M3_TREE_NULL;
        L.userData = shape;
        L.height = 0;
        L.pad = 0;
        PutBound(leaf, mine);
    }
};

#endif // M3_TREEWALK_CUH
